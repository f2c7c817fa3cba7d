// Triangle-listing form of the support product (GA_TRI): C<A> = A·A for a
// symmetric matrix A whose stored values are all 1 — the product the
// reference's k_truss evaluates every iteration (src/main.cpp:103,
// Tmp<C> = C·C) and whose row sums its triangle counts take.
//
// For such an A, C(i, j) = |N(i) ∩ N(j)| over vertices other than i and j
// (the triangles through edge {i, j}), plus 1 for each of i and j that holds
// a diagonal entry; C(i, i) = |N(i)| (the row's length, diagonal included).
// Every triangle is listed once: vertices get ranks 0..m-1 in order of
// degree (a counting sort, once per call; or their indices), each undirected
// edge is kept in the direction of increasing rank (the oriented list O_u of
// u holds the neighbours ranked above u, in column order), and a triangle
// u < v < w (by rank) is found as the wedge u -> v -> w with w in O_u. Its
// three edges' counts are raised: (u, v) by the entry's hit total, (u, w) in
// shared memory, (v, w) by a global atomic. Integer counts: the result is
// exact whatever the order, and whatever order ties of degree get.
//
// Lookups: each warp keeps a bitmap of O_u's members in a window of kTriWin
// ranks ending at O_u's highest rank, with per-word popcount prefixes giving
// a member's index in O(1); a w ranked below the window is binary-searched
// in O_u. Ranked by degree, almost every wedge of a power-law graph ends at
// a vertex of the top ranks (the hubs), inside the window. The ranks may
// also be the vertex indices (GA_OPT_TRI_ORDER): then the lists of a union
// of small graphs span fewer ranks than the window and no search is needed.
//
// A single evaluation (ga_mxm_masked, triangle counting, the autotuner) builds
// separate oriented lists; all launches read the current entry count on the
// device:
//   orient     rank flags per entry, diagonal flags, work counters
//   scan       flags -> positions in the oriented lists
//   scatter    oriented columns and their ranks, zeroed counts, oriented row
//              starts, tasks per row (kTriTask oriented entries each)
//   scan       tasks per row -> task starts; task list
//   support    one warp per task
//   writeback  counts (+ diagonal terms) to both mirror entries; C(i, i)
// The k-truss loop keeps the orientation in C itself instead (the `trikt`
// kernels at the end of this file): every row is stored as [oriented part |
// the rest] for the whole loop, so an iteration is task list, support, keep
// flags and the prune.
#include "ga_device.cuh"
#include "ga_loop.cuh"

#include <algorithm>
#include <cstddef>
#include <cstring>
#include <map>
#include <mutex>

namespace ga {

constexpr int kTriThreads = 128;
constexpr int kTriTask = 16;                  // oriented entries per warp task (at most 32)
constexpr int kTriWin = 1 << 14;              // rank window of the member bitmaps
constexpr int kTriWinWords = kTriWin / 32;    // 512 bitmap words per warp
constexpr int kTriCntMax = 1024;              // longest O_u counted in shared memory
constexpr int kTriCntWords = kTriCntMax / 4;  // byte counters, four per word

// ------------------------------------------------------------------ ranks
// Degrees repeat a lot (a power-law graph has many vertices of degree 0, 1,
// 2, ...), so the lanes of a warp that share a degree are grouped
// (__match_any_sync) and one of them updates the bucket for the group.
__global__ void k_tri_deg_count(const int32_t* __restrict__ cr, int64_t m, int32_t* __restrict__ hist) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); b < m; b += stride) {
        const int64_t v = b + lane;
        const int32_t d = v < m ? cr[v + 1] - cr[v] : -1;
        const unsigned grp = __match_any_sync(0xffffffffu, d);
        if (d >= 0 && lane == __ffs(grp) - 1) atomicAdd(hist + d, __popc(grp));
    }
}

// After the scan of the degree histogram: rank = next free place of the
// vertex's degree bucket (a group of lanes with one degree reserves its
// places with one atomic).
__global__ void k_tri_rank(const int32_t* __restrict__ cr, int64_t m, int32_t* __restrict__ next,
                           int32_t* __restrict__ rank) {
    const int lane = threadIdx.x & 31;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t b = (int64_t)blockIdx.x * blockDim.x + (threadIdx.x & ~31); b < m; b += stride) {
        const int64_t v = b + lane;
        const int32_t d = v < m ? cr[v + 1] - cr[v] : -1;
        const unsigned grp = __match_any_sync(0xffffffffu, d);
        const int leader = __ffs(grp) - 1;
        int32_t base = 0;
        if (d >= 0 && lane == leader) base = atomicAdd(next + d, __popc(grp));
        base = __shfl_sync(0xffffffffu, base, leader);
        if (d >= 0) rank[v] = base + __popc(grp & ((1u << lane) - 1u));
    }
}

// Ranks by degree inside each graph of a batch (rows of graph g: voff[g] ..
// voff[g + 1] - 1): bucket of vertex v. A graph of n vertices has n buckets, so
// its highest one takes degree n too (a diagonal entry in a full row).
__device__ __forceinline__ int32_t tri_graph_bucket(const int32_t* __restrict__ cr, const int32_t* __restrict__ gid,
                                                    const int32_t* __restrict__ voff, int64_t v) {
    const int32_t b = voff[gid[v]], n = voff[gid[v] + 1] - b;
    return b + min(cr[v + 1] - cr[v], n - 1);
}

__global__ void k_tri_graph_deg_count(const int32_t* __restrict__ cr, int64_t m, const int32_t* __restrict__ gid,
                                      const int32_t* __restrict__ voff, int32_t* __restrict__ hist) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < m; v += (int64_t)gridDim.x * blockDim.x)
        atomicAdd(hist + tri_graph_bucket(cr, gid, voff, v), 1);
}

__global__ void k_tri_graph_rank(const int32_t* __restrict__ cr, int64_t m, const int32_t* __restrict__ gid,
                                 const int32_t* __restrict__ voff, int32_t* __restrict__ next,
                                 int32_t* __restrict__ rank) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < m; v += (int64_t)gridDim.x * blockDim.x)
        rank[v] = atomicAdd(next + tri_graph_bucket(cr, gid, voff, v), 1);
}

__global__ void k_tri_iota(int64_t m, int32_t* __restrict__ rank) {
    for (int64_t v = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; v < m; v += (int64_t)gridDim.x * blockDim.x)
        rank[v] = (int32_t)v;
}

// Rank flag of every entry (column ranked above the row: kept in O_row),
// diagonal flags, and the Gustavson work counters the other forms report:
// counts 1, as for a k-truss support that evaluates the upper triangle
// (products of the rows whose upper part is not empty, upper entries); 2, as
// for the whole mask; 0, none (triangle counting).
__global__ void k_tri_orient(const int32_t* __restrict__ cr, const int32_t* __restrict__ cc,
                             const int32_t* __restrict__ row_of, const int32_t* __restrict__ rank, int64_t m,
                             int64_t cap, int32_t* __restrict__ flag, int32_t* __restrict__ diag,
                             unsigned long long* __restrict__ ctr, int counts) {
    const bool upper = counts == 1;
    const int64_t cur = cr[m];
    unsigned long long prod = 0, mask = 0;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < cap; q += (int64_t)gridDim.x * blockDim.x) {
        int32_t f = 0;
        if (q < cur) {
            const int32_t i = row_of[q], j = cc[q];
            if (i == j) diag[i] = 1;
            else f = rank[j] > rank[i];
            if (counts && (!upper || j >= i)) ++mask;
            if (counts && (!upper || cc[cr[i + 1] - 1] >= i)) prod += (unsigned long long)(cr[j + 1] - cr[j]);
        }
        flag[q] = f;
    }
    prod = warp_sum<unsigned long long>(prod);
    mask = warp_sum<unsigned long long>(mask);
    if ((threadIdx.x & 31) == 0) {
        if (prod) atomicAdd(&ctr[GA_CTR_PRODUCTS], prod);
        if (mask) atomicAdd(&ctr[GA_CTR_MASK_ENTRIES], mask);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&ctr[GA_CTR_LAUNCHES], 1ull);
        atomicAdd(&ctr[GA_CTR_A_ENTRIES], (unsigned long long)cur);
        atomicAdd(&ctr[GA_CTR_ROWS], (unsigned long long)m);
    }
}

// After the scan `pos` of the flags: oriented columns, their ranks and
// zeroed counts at their positions, oriented row starts ost[i] = pos[cr[i]],
// and the number of warp tasks of each row.
__global__ void k_tri_scatter(const int32_t* __restrict__ cr, const int32_t* __restrict__ cc,
                              const int32_t* __restrict__ pos, const int32_t* __restrict__ rank, int64_t m,
                              int32_t* __restrict__ ocol, int32_t* __restrict__ orank, int32_t* __restrict__ sup_o,
                              int32_t* __restrict__ ost, int32_t* __restrict__ ntask) {
    const int64_t cur = cr[m];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < cur || q <= m; q += stride) {
        if (q <= m) {
            const int32_t s = pos[cr[q]];
            ost[q] = s;
            if (q < m) ntask[q] = (pos[cr[q + 1]] - s + kTriTask - 1) / kTriTask;
        }
        if (q < cur) {
            const int32_t d = pos[q];
            if (pos[q + 1] != d) {
                const int32_t j = cc[q];
                ocol[d] = j;
                orank[d] = rank[j];
                sup_o[d] = 0;
            }
        }
    }
}

// Row of every task (tasks of row u: tstart[u] .. tstart[u+1]-1).
__global__ void k_tri_tasklist(const int32_t* __restrict__ tstart, int64_t m, int32_t* __restrict__ task_row) {
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < m; u += (int64_t)gridDim.x * blockDim.x)
        for (int32_t t = tstart[u]; t < tstart[u + 1]; ++t) task_row[t] = (int32_t)u;
}

// One warp per task: up to kTriTask consecutive entries (u, v) of O_u
// (O_u = [ost[u], ost[u+1]), or [ost[u], ost[u] + ocnt[u]) with ocnt). The
// warp marks O_u's members of the rank window [win0, win0 + kTriWin) in its
// bitmap (an O_u longer than kTriCntMax uses 32 bucket splitters in
// registers and a short binary search instead). For each entry v in turn,
// the lanes take 32 entries w of O_v at a time: a member is the triangle
// (u, v, w). Its (u, v) count is the entry's ballot total (one atomic per
// entry), (u, w) a byte counter per member in shared memory (added to the
// oriented counts when the task ends; a task adds at most kTriTask to one
// member), (v, w) a global atomic.
//
// COUNT: triangle counting instead: no edge counts; each triangle adds 1 to
// the total and, with per_row, to the row of its largest vertex index (the
// row sums of C<L> = L·L over the strictly lower triangle L). Where that is u
// or v, the entry's hits are added together: one atomic per entry. Only a w
// above both takes one of its own; w has the highest degree of the three, and
// a power-law graph's hubs mostly have low indices. One atomic per triangle
// took 3.32 ms on R-MAT 18, this form 2.35 ms.
template <bool COUNT>
__global__ void __launch_bounds__(kTriThreads, 10) k_tri_support(const int32_t* __restrict__ ost,
                                                             const int32_t* __restrict__ ocnt,
                                                             const int32_t* __restrict__ ocol,
                                                             const int32_t* __restrict__ orank,
                                                             const int32_t* __restrict__ tstart,
                                                             const int32_t* __restrict__ task_row, int64_t m,
                                                             int32_t* __restrict__ sup_o,
                                                             unsigned long long* __restrict__ ctr,
                                                             unsigned long long* __restrict__ total,
                                                             unsigned long long* __restrict__ per_row) {
    // per bitmap word: its member bits (x) and the member index of its first
    // member (y), read together by one 64-bit shared load
    __shared__ uint2 words_s[kTriThreads / 32][kTriWinWords + 1];  // the last: a guard, stays zero
    __shared__ uint32_t cnt_s[kTriThreads / 32][kTriCntWords];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    uint2* words = words_s[threadIdx.x >> 5];
    uint32_t* cnt = cnt_s[threadIdx.x >> 5];
    for (int s = lane; s <= kTriWinWords; s += 32) words[s] = make_uint2(0u, 0u);
    for (int s = lane; s < kTriCntWords; s += 32) cnt[s] = 0;
    __syncwarp();
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int64_t ntask = tstart[m];
    unsigned long long wedges = 0, tris = 0;
    for (int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c < ntask; c += warps) {
        const int u = task_row[c];
        const int32_t ub = ost[u], un = ocnt ? ocnt[u] : ost[u + 1] - ub;
        const int32_t p0 = ub + (int32_t)(c - tstart[u]) * kTriTask;
        const int ne = min(kTriTask, ub + un - p0);
        const int32_t* Ou = ocol + ub;
        const bool counted = un <= kTriCntMax;
        // the task's entries (u, v) and v's lists, loaded before the bitmap
        // is built so the two chains of loads overlap
        int32_t v = 0, vs = 0, vn = 0;
        if (lane < ne) {
            v = __ldg(ocol + p0 + lane);
            vs = __ldg(ost + v);
            vn = ocnt ? __ldg(ocnt + v) : __ldg(ost + v + 1) - vs;
        }
        int32_t key = 0;
        int n_in = 0;
        // window: the kTriWin ranks up to O_u's highest (all of O_u when its
        // ranks span fewer); members below it are binary-searched
        int32_t win0 = 0;
        int nwords = 0;  // bitmap words the members span
        bool below = false;
        if (counted) {
            int32_t lo = INT32_MAX, hi = -1;
            for (int t = lane; t < un; t += 32) {
                const int32_t r = __ldg(orank + ub + t);
                lo = min(lo, r);
                hi = max(hi, r);
            }
            lo = __reduce_min_sync(FULL, lo);
            hi = __reduce_max_sync(FULL, hi);
            win0 = max(lo, hi - kTriWin + 1);
            below = lo < win0;
            nwords = ((hi - win0) >> 5) + 1;
            for (int t = lane; t < un; t += 32) {
                const int32_t b = __ldg(orank + ub + t) - win0;
                if (b >= 0) atomicOr(&words[b >> 5].x, 1u << (b & 31));
            }
            __syncwarp();
        }
        if (counted && !COUNT) {
            // member index of the first member of every bitmap word
            int run = 0;
            for (int k = 0; k < nwords; k += 32) {
                const int c1 = __popc(words[k + lane].x);
                const int incl = warp_incl_scan(c1);
                words[k + lane].y = (uint32_t)(run + incl - c1);
                run += __shfl_sync(FULL, incl, 31);
            }
            n_in = run;
            __syncwarp();
        } else if (!counted) {
            key = __ldg(Ou + (int)(((int64_t)(lane + 1) * un) >> 5) - 1);
        }
        for (int e = 0; e < ne; ++e) {
            const int32_t evs = __shfl_sync(FULL, vs, e);
            const int32_t evn = __shfl_sync(FULL, vn, e);
            const int32_t ev = __shfl_sync(FULL, v, e);
            uint32_t mine = 0;  // this lane's hits for the entry
            uint32_t own = 0;   // of those, the ones that the row max(u, v) takes
            const int32_t top = max(u, ev);
            // one round of 32 wedges: the lane's wedge x of the entry, ld its
            // loaded rank (column when the list is not counted); INT32_MAX
            // past the list's end, which no lookup matches
            auto probe = [&](int32_t x, int32_t ld) {
                const int32_t wp = evs + x;
                bool hit = false;
                if (counted) {
                    // the word moved up so that w's bit is its sign, and what
                    // is below it the member index; ranks outside the window
                    // read the guard (those above it are above every member).
                    // A range check, a shift and two masks instead: 46M
                    // entries of 30-NN graphs 3.43 ms, so 3.26
                    const uint32_t b = min((uint32_t)(ld - win0), (uint32_t)kTriWin);
                    const uint2 wd = words[b >> 5];
                    const uint32_t up = __funnelshift_l(0u, wd.x, ~b);
                    if ((int32_t)up < 0) {
                        hit = true;
                        if (!COUNT) {
                            const int idx = (int)wd.y + __popc(up) - 1;
                            atomicAdd(cnt + (idx >> 2), 1u << ((idx & 3) << 3));  // (u, w)
                        }
                    } else if (below && ld < win0) {
                        // below the window: binary search of O_u by column
                        const int32_t w = __ldg(ocol + wp);
                        const int t = lower_bound_i32(Ou, un, w);
                        if (t < un && __ldg(Ou + t) == w) {
                            hit = true;
                            if (!COUNT) atomicAdd(sup_o + ub + t, 1);  // (u, w)
                        }
                    }
                } else {
                    const int32_t w = ld;
                    const int bb = warp_lower_bound(key, w);
                    if (bb < 32) {
                        const int lo_b = (int)(((int64_t)bb * un) >> 5);
                        const int hi_b = (int)(((int64_t)(bb + 1) * un) >> 5);
                        const int t = lo_b + lower_bound_i32(Ou + lo_b, hi_b - lo_b, w);
                        if (t < hi_b && __ldg(Ou + t) == w) {
                            hit = true;
                            if (!COUNT) atomicAdd(sup_o + ub + t, 1);  // (u, w)
                        }
                    }
                }
                if (!COUNT && hit) atomicAdd(sup_o + wp, 1);  // (v, w)
                if (COUNT && hit && per_row) {
                    const int32_t w = __ldg(ocol + wp);
                    if (w > top) atomicAdd(per_row + w, 1ull);
                    else ++own;
                }
                mine += hit ? 1u : 0u;
            };
            // two rounds per pass, both loads issued first
            const int32_t* src = counted ? orank : ocol;
            for (int32_t base = 0; base < evn; base += 64) {
                const int32_t x0 = base + lane, x1 = x0 + 32;
                const int32_t l0 = x0 < evn ? __ldg(src + evs + x0) : INT32_MAX;
                const int32_t l1 = x1 < evn ? __ldg(src + evs + x1) : INT32_MAX;
                probe(x0, l0);
                if (base + 32 < evn) probe(x1, l1);  // warp-uniform
            }
            const int32_t found = (int32_t)__reduce_add_sync(FULL, mine);
            if (lane == 0) {
                wedges += (unsigned long long)evn;
                tris += (unsigned long long)found;
                if (!COUNT && found) atomicAdd(sup_o + p0 + e, found);  // (u, v)
            }
            if (COUNT && per_row && found) {  // warp-uniform
                own = __reduce_add_sync(FULL, own);
                if (lane == 0 && own) atomicAdd(per_row + top, (unsigned long long)own);
            }
        }
        if (counted && COUNT) {
            __syncwarp();
            for (int s = lane; s < nwords; s += 32) words[s] = make_uint2(0u, 0u);
            __syncwarp();
        } else if (counted) {
            __syncwarp();
            for (int t = lane; t < un; t += 32) {
                const int32_t b = __ldg(orank + ub + t) - win0;
                if (b >= 0) {
                    const uint2 wd = words[b >> 5];
                    const int idx = (int)wd.y + __popc(wd.x & ((1u << (b & 31)) - 1u));
                    const uint32_t n = (cnt[idx >> 2] >> ((idx & 3) * 8)) & 0xffu;
                    if (n) atomicAdd(sup_o + ub + t, (int32_t)n);
                }
            }
            __syncwarp();
            for (int s = lane; s < nwords; s += 32) words[s] = make_uint2(0u, 0u);
            for (int s = lane; s < ((n_in + 3) >> 2); s += 32) cnt[s] = 0;
            __syncwarp();
        }
    }
    if (lane == 0) {
        if (wedges) atomicAdd(&ctr[GA_CTR_WEDGES], wedges);
        if (tris) atomicAdd(&ctr[GA_CTR_TRIANGLES], tris);
        if (COUNT && tris) atomicAdd(total, tris);
    }
}

// Support of every entry of C: an oriented entry's count plus the diagonal
// terms goes to it and to its mirror; a diagonal entry gets its row length.
__global__ void k_tri_writeback(const int32_t* __restrict__ cr, const int32_t* __restrict__ cc,
                                const int32_t* __restrict__ row_of, const int32_t* __restrict__ mir,
                                const int32_t* __restrict__ pos, const int32_t* __restrict__ sup_o,
                                const int32_t* __restrict__ diag, int64_t m, int32_t* __restrict__ sup) {
    const int64_t cur = cr[m];
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < cur; q += (int64_t)gridDim.x * blockDim.x) {
        const int32_t i = row_of[q], j = cc[q];
        if (i == j) {
            sup[q] = cr[i + 1] - cr[i];
            continue;
        }
        const int32_t d = pos[q];
        if (pos[q + 1] != d) {
            const int32_t s = sup_o[d] + diag[i] + diag[j];
            sup[q] = s;
            sup[mir[q]] = s;
        }
    }
}

static size_t align256(size_t b) { return (b + 255) & ~(size_t)255; }

namespace {
struct TriScratch {
    int32_t *ocol, *orank, *sup_o, *task_row, *ost, *tstart, *diag, *rank;
    void* scan_scr;
};

size_t task_cap(int64_t m, int64_t cap) { return (size_t)(cap / kTriTask + m + 1); }

// Carves the buffers out of `scratch` (nullptr: only sizes them); returns
// the bytes used.
size_t carve(void* scratch, int64_t m, int64_t cap, TriScratch* t) {
    const size_t c = (size_t)(cap > 0 ? cap : 1), r = (size_t)m + 2;
    unsigned char* base = static_cast<unsigned char*>(scratch);
    size_t off = 0;
    auto take = [&](size_t count) {
        int32_t* p = base ? reinterpret_cast<int32_t*>(base + off) : nullptr;
        off += align256(sizeof(int32_t) * count);
        return p;
    };
    TriScratch s;
    s.ocol = take(c);
    s.orank = take(c);
    s.sup_o = take(c);
    s.task_row = take(task_cap(m, cap));
    s.ost = take(r);
    s.tstart = take(r);
    s.diag = take(r);
    s.rank = take(r);
    s.scan_scr = base ? base + off : nullptr;
    off += align256(scan_scratch_bytes((cap > m ? cap : m) + 2));
    if (t) *t = s;
    return off;
}
}  // namespace

size_t tri_scratch_bytes(int64_t m, int64_t cap) { return carve(nullptr, m, cap, nullptr); }

void tri_prepare(ga_ctx ctx, ga_csr C, void* scratch, int64_t cap) {
    const int64_t m = C->m;
    if (m == 0) return;
    TriScratch t;
    carve(scratch, m, cap, &t);
    const int grid = grid_for(m, 256, ctx->num_sms * 8);
    if (ctx->tune.tri_order == 1) {  // index order
        k_tri_iota<<<grid, 256, 0, ctx->stream>>>(m, t.rank);
        post_launch("tri_iota");
        return;
    }
    // ranks by degree: histogram of the degrees (0..m), its scan, then each
    // vertex takes the next place of its degree's bucket
    int32_t* hist = t.tstart;
    GA_CUDA(cudaMemsetAsync(hist, 0, sizeof(int32_t) * (size_t)(m + 2), ctx->stream));
    k_tri_deg_count<<<grid, 256, 0, ctx->stream>>>(C->rst, m, hist);
    post_launch("tri_deg_count");
    scan_exclusive_i32_scratch(ctx, hist, hist, m + 1, t.scan_scr);
    k_tri_rank<<<grid, 256, 0, ctx->stream>>>(C->rst, m, hist, t.rank);
    post_launch("tri_rank");
}

// Orientation, oriented lists and the task list of C's current pattern.
static void tri_lists(ga_ctx ctx, ga_csr C, const int32_t* row_of, int32_t* pos, const TriScratch& t, int64_t cap,
                      int counts) {
    const int64_t m = C->m;
    const int grid_ent = grid_for(cap, 256, ctx->num_sms * 16);
    const int grid_copy = grid_for(m + cap, 256, ctx->num_sms * 8);
    const int grid_rows = grid_for(m, 256, ctx->num_sms * 8);
    ProfScope ps(ctx, "tri_orient");
    GA_CUDA(cudaMemsetAsync(t.diag, 0, sizeof(int32_t) * (size_t)m, ctx->stream));
    k_tri_orient<<<grid_ent, 256, 0, ctx->stream>>>(C->rst, C->col, row_of, t.rank, m, cap, pos, t.diag,
                                                    ctx->d_counters, counts);
    post_launch("tri_orient");
    scan_exclusive_i32_scratch(ctx, pos, pos, cap, t.scan_scr);
    k_tri_scatter<<<grid_copy, 256, 0, ctx->stream>>>(C->rst, C->col, pos, t.rank, m, t.ocol, t.orank, t.sup_o,
                                                      t.ost, t.tstart);
    post_launch("tri_scatter");
    scan_exclusive_i32_scratch(ctx, t.tstart, t.tstart, m, t.scan_scr);
    k_tri_tasklist<<<grid_rows, 256, 0, ctx->stream>>>(t.tstart, m, t.task_row);
    post_launch("tri_tasklist");
}

// Persistent grid: as many blocks as are resident at once.
template <bool COUNT>
static int tri_blocks_per_sm() {
    static const int per_sm = [] {
        int b = 0;
        if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&b, k_tri_support<COUNT>, kTriThreads, 0) != cudaSuccess ||
            b < 1)
            b = 1;
        return b;
    }();
    return per_sm;
}

void tri_support_launch(ga_ctx ctx, ga_csr C, const int32_t* row_of, const int32_t* mir, int32_t* pos,
                        int32_t* sup, void* scratch, int64_t cap, bool upper_counts) {
    const int64_t m = C->m;
    if (m == 0) return;
    TriScratch t;
    carve(scratch, m, cap, &t);
    tri_lists(ctx, C, row_of, pos, t, cap, upper_counts ? 1 : 2);
    {
        ProfScope ps(ctx, "tri_support");
        k_tri_support<false><<<ctx->num_sms * tri_blocks_per_sm<false>(), kTriThreads, 0, ctx->stream>>>(
            t.ost, nullptr, t.ocol, t.orank, t.tstart, t.task_row, m, t.sup_o, ctx->d_counters, nullptr, nullptr);
        post_launch("tri_support");
    }
    ProfScope ps(ctx, "tri_writeback");
    k_tri_writeback<<<grid_for(cap, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(C->rst, C->col, row_of, mir,
                                                                                   pos, t.sup_o, t.diag, m, sup);
    post_launch("tri_writeback");
}

void tri_count(ga_ctx ctx, ga_csr A, unsigned long long* d_total, unsigned long long* d_per_row) {
    const int64_t m = A->m, cap = A->nnz;
    if (d_per_row) GA_CUDA(cudaMemsetAsync(d_per_row, 0, sizeof(int64_t) * (size_t)m, ctx->stream));
    if (m == 0 || cap == 0) return;
    DBuf<int32_t> row_of(ctx, (size_t)cap), pos(ctx, (size_t)cap + 1);
    DBuf<unsigned char> scr(ctx, tri_scratch_bytes(m, cap));
    TriScratch t;
    carve(scr.p, m, cap, &t);
    expand_rows(ctx, A, row_of.p);
    tri_prepare(ctx, A, scr.p, cap);
    tri_lists(ctx, A, row_of.p, pos.p, t, cap, 0);
    ProfScope ps(ctx, "tri_count");
    k_tri_support<true><<<ctx->num_sms * tri_blocks_per_sm<true>(), kTriThreads, 0, ctx->stream>>>(
        t.ost, nullptr, t.ocol, t.orank, t.tstart, t.task_row, m, nullptr, ctx->d_counters, d_total, d_per_row);
    post_launch("tri_count");
}

bool tri_applies(ga_ctx ctx, ga_csr A, ga_csr B, ga_csr M) {
    const bool same = (A == B || (A->rst == B->rst && A->col == B->col && A->val == B->val)) &&
                      (A == M || (A->rst == M->rst && A->col == M->col));
    return same && A->dtype == GA_INT32 && csr_is_symmetric(ctx, A) && csr_unit_values(ctx, A);
}

// C<A> = A·A by triangle listing into values aligned with A's pattern.
void tri_masked_into(ga_ctx ctx, ga_csr A, int32_t* sup) {
    const int64_t m = A->m, cap = A->nnz;
    if (m == 0 || cap == 0) return;
    DBuf<int32_t> row_of(ctx, (size_t)cap), mir(ctx, (size_t)cap), pos(ctx, (size_t)cap + 1);
    DBuf<unsigned char> scr(ctx, tri_scratch_bytes(m, cap));
    expand_rows(ctx, A, row_of.p);
    mirror_index(ctx, A, row_of.p, mir.p);
    tri_prepare(ctx, A, scr.p, cap);
    tri_support_launch(ctx, A, row_of.p, mir.p, pos.p, sup, scr.p, cap, false);
}

// =============================================== resident orientation (k-truss)
// Ranks of flagged entries. A flag takes one bit of a 32-entry word, and the
// words' counts are scanned, not the entries: a 32nd of the scan's work, and
// a rank is read from two small arrays (R-MAT 18, 7.6M entries: flags, scan
// and placing 124 us with an int per entry, 92 with words).
struct WordRanks {
    uint32_t* bits;  // word w: entries 32 w ..
    int32_t* pre;    // flags before word w; the last word's next holds their number
};
// Flagged entries before entry q (q: up to the number of entries).
__device__ __forceinline__ int32_t word_rank(const WordRanks& r, int64_t q) {
    return r.pre[q >> 5] + __popc(r.bits[q >> 5] & ((1u << (q & 31)) - 1u));
}
__device__ __forceinline__ bool word_flag(const WordRanks& r, int64_t q) { return r.bits[q >> 5] >> (q & 31) & 1u; }
// Words that word_rank reads for q <= entries.
static int64_t rank_words(int64_t entries) { return entries / 32 + 1; }

// Entry q of the unpartitioned C (column order) goes to the oriented part of
// its row when its column is ranked above the row. One warp per word.
__global__ void k_trikt_part_flags(const int32_t* __restrict__ cc, const int32_t* __restrict__ row_of,
                                   const int32_t* __restrict__ rank, int64_t nnz, WordRanks r) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5), words = nnz / 32 + 1;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < words; w += warps) {
        const int64_t q = w * 32 + lane;
        bool f = false;
        if (q < nnz) {
            const int32_t i = row_of[q], j = cc[q];
            f = i != j && rank[j] > rank[i];
        }
        const unsigned b = __ballot_sync(0xffffffffu, f);
        if (lane == 0) {
            r.bits[w] = b;
            r.pre[w] = __popc(b);
        }
    }
}

// Place of entry q of row [rb, re) in the stable partition of the row.
__device__ __forceinline__ int32_t part_place(const WordRanks& r, int64_t q, int32_t rb, int32_t oc, bool* oriented) {
    const int32_t before = word_rank(r, q) - word_rank(r, rb);  // oriented entries before q in its row
    *oriented = word_flag(r, q);
    return *oriented ? rb + before : rb + oc + (int32_t)(q - rb) - before;
}

// After the scan: the partition of every row (oriented part, then the rest),
// the rank of every placed column, and per row its oriented count and tasks
// (its diagonal position comes later).
__global__ void k_trikt_part_place(const int32_t* __restrict__ cr, const int32_t* __restrict__ cc,
                                   const int32_t* __restrict__ row_of, const int32_t* __restrict__ rank, WordRanks r,
                                   int64_t m, int64_t nnz, int32_t* __restrict__ out_col,
                                   int32_t* __restrict__ crank, int32_t* __restrict__ ocount,
                                   int32_t* __restrict__ ntask, int32_t* __restrict__ dpos) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nnz || q < m; q += stride) {
        if (q < m) {
            dpos[q] = -1;
            const int32_t oc = word_rank(r, cr[q + 1]) - word_rank(r, cr[q]);
            ocount[q] = oc;
            ntask[q] = (oc + kTriTask - 1) / kTriTask;
        }
        if (q < nnz) {
            const int32_t i = row_of[q], rb = cr[i], j = cc[q];
            bool o;
            const int32_t np = part_place(r, q, rb, word_rank(r, cr[i + 1]) - word_rank(r, rb), &o);
            out_col[np] = j;
            crank[np] = rank[j];
        }
    }
}

// Mirror of every entry and each row's diagonal position in the partitioned
// layout: (j, i) lies in the oriented part of row j when i is ranked above j.
__global__ void k_trikt_part_mirror(const int32_t* __restrict__ cr, const int32_t* __restrict__ cc,
                                    const int32_t* __restrict__ row_of, const int32_t* __restrict__ crank,
                                    const int32_t* __restrict__ ocount, int64_t nnz, int32_t* __restrict__ mir,
                                    int32_t* __restrict__ dpos) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nnz; q += (int64_t)gridDim.x * blockDim.x) {
        const int32_t i = row_of[q], j = cc[q];
        if (i == j) {
            dpos[i] = (int32_t)q;
            mir[q] = (int32_t)q;
            continue;
        }
        // rank of i: the mirror's rank; q is oriented in row i iff rank(j) > rank(i)
        const bool q_oriented = (int64_t)q - cr[i] < ocount[i];
        const int32_t b = q_oriented ? cr[j] + ocount[j] : cr[j];  // i ranks below j: the rest of row j
        const int32_t e = q_oriented ? cr[j + 1] : cr[j] + ocount[j];
        mir[q] = b + lower_bound_i32(cc + b, e - b, i);
    }
}

// Keep flags: an oriented entry's support is its count, another entry's the
// count of its mirror (plus one per diagonal entry of its two rows); a
// diagonal entry's support is its row's length. Work counters as for an
// upper-triangle support product.
__global__ void k_trikt_flags(const int32_t* __restrict__ cr, const int32_t* __restrict__ cc,
                              const int32_t* __restrict__ row_of, const int32_t* __restrict__ mir,
                              const int32_t* __restrict__ ocount, const int32_t* __restrict__ dpos,
                              const int32_t* __restrict__ sup, int64_t m, int64_t cap, int k,
                              const int32_t* __restrict__ gid, const int32_t* __restrict__ done_g,
                              const int32_t* __restrict__ kg, int32_t* __restrict__ flag,
                              unsigned long long* __restrict__ ctr) {
    const int64_t cur = cr[m];
    unsigned long long prod = 0, mask = 0;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < cap; q += (int64_t)gridDim.x * blockDim.x) {
        int32_t keep = 0;
        if (q < cur) {
            const int32_t i = row_of[q], j = cc[q];
            const int32_t rb = cr[i], re = cr[i + 1], oc = ocount[i];
            int32_t s;
            if (i == j) s = re - rb;
            else s = sup[q - rb < oc ? q : mir[q]] + (dpos[i] >= 0) + (dpos[j] >= 0);
            if (kg) {
                const int g = gid[i];
                keep = done_g[g] != 0 || s >= kg[g] - 2;
            } else {
                keep = s >= k - 2;
                if (!keep && gid) keep = done_g[gid[i]] != 0;
            }
            // the row's largest column: the last of either part
            const int32_t cmax = max(oc > 0 ? cc[rb + oc - 1] : -1, re > rb + oc ? cc[re - 1] : -1);
            if (j >= i) ++mask;
            if (cmax >= i) prod += (unsigned long long)(cr[j + 1] - cr[j]);
        }
        flag[q] = keep;
    }
    prod = warp_sum<unsigned long long>(prod);
    mask = warp_sum<unsigned long long>(mask);
    if ((threadIdx.x & 31) == 0) {
        if (prod) atomicAdd(&ctr[GA_CTR_PRODUCTS], prod);
        if (mask) atomicAdd(&ctr[GA_CTR_MASK_ENTRIES], mask);
    }
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&ctr[GA_CTR_LAUNCHES], 1ull);
        atomicAdd(&ctr[GA_CTR_A_ENTRIES], (unsigned long long)cur);
        atomicAdd(&ctr[GA_CTR_ROWS], (unsigned long long)m);
    }
}

// After the flags' scan: kept entries move to pos[q] (columns, rows, column
// ranks), pos_new[q] is the new position or -1, the new row starts are
// tr[i] = pos[cr[i]]; per row the oriented count shrinks to the kept
// oriented entries (updated in place: unchanged when nothing was pruned) and
// the next iteration's task count follows.
__global__ void k_trikt_scatter(const int32_t* __restrict__ cr, const int32_t* __restrict__ cc,
                                const int32_t* __restrict__ pos, const int32_t* __restrict__ row_of,
                                const int32_t* __restrict__ crank, int64_t m, int32_t* __restrict__ ocount,
                                int32_t* __restrict__ ntask, int32_t* __restrict__ tc, int32_t* __restrict__ tr,
                                int32_t* __restrict__ pos_new, int32_t* __restrict__ trow,
                                int32_t* __restrict__ tcrank, const int32_t* __restrict__ gid,
                                const int32_t* __restrict__ done_g) {
    const int64_t cur = cr[m];
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < cur || q <= m; q += stride) {
        if (q <= m) {
            tr[q] = pos[cr[q]];
            if (q < m) {
                const int32_t rb = cr[q];
                const int32_t oc = pos[rb + ocount[q]] - pos[rb];
                ocount[q] = oc;
                // rows of finished graphs (batches) need no more support
                ntask[q] = gid && done_g[gid[q]] ? 0 : (oc + kTriTask - 1) / kTriTask;
            }
        }
        if (q < cur) {
            const int32_t d = pos[q];
            const bool keep = pos[q + 1] != d;
            if (keep) {
                tc[d] = cc[q];
                trow[d] = row_of[q];
                tcrank[d] = crank[q];
            }
            pos_new[q] = keep ? d : -1;
        }
    }
}

// When the iteration swapped: C <- the pruned matrix (row starts, columns,
// values 1), and the per-entry arrays (rows, mirrors, column ranks) and the
// diagonal positions follow it; one launch for all of them.
__global__ void k_trikt_copyback(const KtState* st, int64_t m, const int32_t* __restrict__ tr,
                                 const int32_t* __restrict__ tc, const int32_t* __restrict__ trow,
                                 const int32_t* __restrict__ mir_new, const int32_t* __restrict__ pos_new,
                                 const int32_t* __restrict__ tcrank, int32_t* __restrict__ cr,
                                 int32_t* __restrict__ cc, int32_t* __restrict__ cv, int32_t* __restrict__ row_of,
                                 int32_t* __restrict__ mir, int32_t* __restrict__ crank,
                                 int32_t* __restrict__ dpos) {
    if (!st->swapped) return;
    const int64_t nnz = st->nnz;
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nnz || q <= m; q += stride) {
        if (q <= m) cr[q] = tr[q];
        if (q < m && dpos[q] >= 0) dpos[q] = pos_new[dpos[q]];
        if (q < nnz) {
            cc[q] = tc[q];
            cv[q] = 1;
            row_of[q] = trow[q];
            mir[q] = mir_new[q];
            crank[q] = tcrank[q];
        }
    }
}

// Rows back in column order: an entry's place in its row is its index in its
// part plus the entries of the other part with smaller columns.
__global__ void k_trikt_unpart(const int32_t* __restrict__ cr, const int32_t* __restrict__ cc,
                               const int32_t* __restrict__ row_of, const int32_t* __restrict__ ocount, int64_t nnz,
                               int32_t* __restrict__ out_col) {
    for (int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; q < nnz; q += (int64_t)gridDim.x * blockDim.x) {
        const int32_t i = row_of[q], rb = cr[i], re = cr[i + 1], oc = ocount[i];
        const int32_t k = (int32_t)(q - rb);
        const bool o = k < oc;
        const int32_t ob = o ? rb + oc : rb, oe = o ? re : rb + oc;
        const int32_t j = cc[q];
        out_col[rb + (o ? k : k - oc) + lower_bound_i32(cc + ob, oe - ob, j)] = j;
    }
}

namespace {
size_t trikt_carve(void* scratch, int64_t m, int64_t cap, TriKt* t) {
    const size_t c = (size_t)(cap > 0 ? cap : 1), r = (size_t)m + 2;
    unsigned char* base = static_cast<unsigned char*>(scratch);
    size_t off = 0;
    auto take = [&](size_t count) {
        int32_t* p = base ? reinterpret_cast<int32_t*>(base + off) : nullptr;
        off += align256(sizeof(int32_t) * count);
        return p;
    };
    TriKt s;
    s.crank = take(c);
    s.tcrank = take(c);
    s.ocount = take(r);
    s.tstart = take(r);
    s.task_row = take(task_cap(m, cap));
    s.dpos = take(r);
    s.rank = take(r);
    s.bits = reinterpret_cast<uint32_t*>(take((size_t)rank_words(cap)));
    s.pre = take((size_t)rank_words(cap) + 1);
    s.scan_scr = base ? base + off : nullptr;
    off += align256(scan_scratch_bytes((cap > m ? cap : m) + 2));
    if (t) *t = s;
    return off;
}
}  // namespace

size_t tri_kt_bytes(int64_t m, int64_t cap) { return trikt_carve(nullptr, m, cap, nullptr); }

void tri_kt_carve(void* scratch, int64_t m, int64_t cap, TriKt* t) { trikt_carve(scratch, m, cap, t); }

// Ranks, and the stable partition of every row of (rst, col) into out_col.
static void trikt_partition(ga_ctx ctx, const int32_t* rst, const int32_t* col, int64_t m, int64_t nnz,
                            const int32_t* row_of, const TriKt& t, const KtBatch* batch, int32_t* out_col) {
    int32_t* rank = t.rank;  // by degree (or index)
    const int grid_v = grid_for(m, 256, ctx->num_sms * 8);
    if (ctx->tune.tri_order == 1) {
        k_tri_iota<<<grid_v, 256, 0, ctx->stream>>>(m, rank);
        post_launch("tri_iota");
    } else if (batch) {
        // A batch ranks each graph's vertices among themselves: by degree over
        // the whole union, a graph's lists span far more ranks than the
        // bitmap window, and most lookups become binary searches. 512 30-NN
        // graphs of up to 4,096 vertices (46M entries): the listing takes
        // 3.40 ms, 6.61 ms with the union's ranks.
        GA_CUDA(cudaMemsetAsync(t.tstart, 0, sizeof(int32_t) * (size_t)(m + 2), ctx->stream));
        k_tri_graph_deg_count<<<grid_v, 256, 0, ctx->stream>>>(rst, m, batch->gid, batch->voff, t.tstart);
        post_launch("tri_deg_count");
        scan_exclusive_i32_scratch(ctx, t.tstart, t.tstart, m, t.scan_scr);
        k_tri_graph_rank<<<grid_v, 256, 0, ctx->stream>>>(rst, m, batch->gid, batch->voff, t.tstart, rank);
        post_launch("tri_rank");
    } else {
        GA_CUDA(cudaMemsetAsync(t.tstart, 0, sizeof(int32_t) * (size_t)(m + 2), ctx->stream));
        k_tri_deg_count<<<grid_v, 256, 0, ctx->stream>>>(rst, m, t.tstart);
        post_launch("tri_deg_count");
        scan_exclusive_i32_scratch(ctx, t.tstart, t.tstart, m + 1, t.scan_scr);
        k_tri_rank<<<grid_v, 256, 0, ctx->stream>>>(rst, m, t.tstart, rank);
        post_launch("tri_rank");
    }
    const WordRanks r{t.bits, t.pre};
    const int64_t words = rank_words(nnz);
    k_trikt_part_flags<<<grid_for(words * 32, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(col, row_of, rank, nnz,
                                                                                            r);
    post_launch("trikt_part_flags");
    scan_exclusive_i32_scratch(ctx, t.pre, t.pre, words, t.scan_scr);
    k_trikt_part_place<<<grid_for(nnz > m ? nnz : m, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(
        rst, col, row_of, rank, r, m, nnz, out_col, t.crank, t.ocount, t.tstart, t.dpos);
    post_launch("trikt_part_place");
}

void tri_kt_setup(ga_ctx ctx, ga_csr C, const int32_t* row_of, int32_t* mir, int32_t* tmp_col, const TriKt& t,
                  const KtBatch* batch) {
    const int64_t m = C->m, nnz = C->nnz;
    trikt_partition(ctx, C->rst, C->col, m, nnz, row_of, t, batch, tmp_col);
    if (nnz) GA_CUDA(cudaMemcpyAsync(C->col, tmp_col, sizeof(int32_t) * (size_t)nnz, cudaMemcpyDeviceToDevice,
                                     ctx->stream));
    if (nnz) {
        k_trikt_part_mirror<<<grid_for(nnz, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(
            C->rst, C->col, row_of, t.crank, t.ocount, nnz, mir, t.dpos);
        post_launch("trikt_part_mirror");
    }
}

void tri_kt_support(ga_ctx ctx, ga_csr C, int32_t* sup, const TriKt& t, int64_t cap) {
    const int64_t m = C->m;
    {
        ProfScope ps(ctx, "tri_orient");
        GA_CUDA(cudaMemsetAsync(sup, 0, sizeof(int32_t) * (size_t)cap, ctx->stream));
        scan_exclusive_i32_scratch(ctx, t.tstart, t.tstart, m, t.scan_scr);
        k_tri_tasklist<<<grid_for(m, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(t.tstart, m, t.task_row);
        post_launch("tri_tasklist");
    }
    ProfScope ps(ctx, "tri_support");
    k_tri_support<false><<<ctx->num_sms * tri_blocks_per_sm<false>(), kTriThreads, 0, ctx->stream>>>(
        C->rst, t.ocount, C->col, t.crank, t.tstart, t.task_row, m, sup, ctx->d_counters, nullptr, nullptr);
    post_launch("tri_support");
}

void tri_kt_flags(ga_ctx ctx, ga_csr C, const int32_t* row_of, const int32_t* mir, const int32_t* sup,
                  const TriKt& t, int64_t cap, int k, const KtBatch* batch, int32_t* flag) {
    k_trikt_flags<<<grid_for(cap, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(
        C->rst, C->col, row_of, mir, t.ocount, t.dpos, sup, C->m, cap, k, batch ? batch->gid : nullptr,
        batch ? batch->done_g : nullptr, batch ? batch->kg : nullptr, flag, ctx->d_counters);
    post_launch("trikt_flags");
}

void tri_kt_scatter(ga_ctx ctx, ga_csr C, const int32_t* pos, const int32_t* row_of, const TriKt& t, int64_t cap,
                    int32_t* tc, int32_t* tr, int32_t* pos_new, int32_t* trow, const KtBatch* batch) {
    k_trikt_scatter<<<grid_for(C->m + cap, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(
        C->rst, C->col, pos, row_of, t.crank, C->m, t.ocount, t.tstart, tc, tr, pos_new, trow, t.tcrank,
        batch ? batch->gid : nullptr, batch ? batch->done_g : nullptr);
    post_launch("trikt_scatter");
}

void tri_kt_copyback(ga_ctx ctx, ga_csr C, const KtState* st, const int32_t* tr, const int32_t* tc,
                     const int32_t* trow, const int32_t* mir_new, const int32_t* pos_new, int32_t* row_of,
                     int32_t* mir, const TriKt& t, int64_t cap) {
    k_trikt_copyback<<<grid_for(C->m + cap, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(
        st, C->m, tr, tc, trow, mir_new, pos_new, t.tcrank, C->rst, C->col, static_cast<int32_t*>(C->val), row_of,
        mir, t.crank, t.dpos);
    post_launch("trikt_copyback");
}

void tri_kt_finish(ga_ctx ctx, ga_csr C, const int32_t* row_of, const TriKt& t, int32_t* tmp_col) {
    const int64_t nnz = C->nnz;
    if (nnz == 0) return;
    k_trikt_unpart<<<grid_for(nnz, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(C->rst, C->col, row_of, t.ocount,
                                                                                   nnz, tmp_col);
    post_launch("trikt_unpart");
    GA_CUDA(cudaMemcpyAsync(C->col, tmp_col, sizeof(int32_t) * (size_t)nnz, cudaMemcpyDeviceToDevice, ctx->stream));
}

// ======================================== frontier k-truss (one matrix)
// The reference's k_truss recomputes the whole support every iteration
// (src/main.cpp:100-127). Between iterations only the triangles that lose
// an edge change, so after one listing the loop keeps the supports and, per
// iteration t with C_t its edges and s_t their exact supports:
//   F_t  = edges of C_t with s_t < k - 2 (iteration 0: found by one pass over
//          the entries; later: the edges whose support crossed below k - 2
//          in iteration t - 1, which are exactly the ones below it);
//   every triangle of C_t with an edge in F_t is destroyed: each of its edges
//          outside F_t loses 1, counted once by the triangle's F_t edge with
//          the smallest id (the position of its oriented entry); an entry
//          (i, i) in F_t lowers every edge of row i by 1 instead, and an edge
//          in F_t shortens its two rows, which lowers their diagonal entries;
//   C_{t+1} = C_t minus F_t; stop when F_t is empty (iteration count t + 1)
//          or after m iterations (count 0), as the reference does.
// Entries never move during the loop: an edge lives at its oriented entry
// (state alive / in F_t / gone, support), the other entry points to it
// (oid); one compaction at the end writes the kept entries in column order.
// A pruned edge's triangles are found by walking the shorter of its two rows
// and binary-searching the other (in the part its rank selects), stopping
// once its support's worth of triangles is found.
//
// Work counters: iteration t adds the Gustavson products of the reference's
// Tmp<C> = C_t*C_t over the rows with an upper part, P_t = sum over entries
// (i, j) of C_t of h(i) deg(j) (h(i): row i has a column >= i; deg: row
// lengths) = sum_j deg(j) H(j), H(j) = entries (i, j) with h(i) = 1. P is
// kept as a running total: an iteration changes deg and H only at the
// endpoints of its pruned edges and, when a row loses its last upper entry
// (once per row and call), at that row's remaining neighbours; those
// vertices' terms are recomputed, so no iteration passes over all entries.
namespace {

enum : uint8_t { kAlive = 0, kDying = 1, kGone = 2 };

struct TriFrontState {
    int32_t cnt[2];              // frontier sizes; the current one is cnt[t & 1]
    int32_t t;                   // iteration
    int32_t done;
    int32_t ntouch;              // vertices whose terms of P change this iteration
    int32_t nflip;               // rows that lost their last upper entry
    int32_t nseg;                // segments of long rows listed this iteration
    uint32_t blocks_done;        // delta kernel: blocks finished
    uint32_t blocks_done_g;      // graph kernel (batches): blocks finished
    // one-launch loop (k_trif_loop); [4]: by iteration
    int32_t nfront[4];           // frontier
    int32_t nt[4], nf[4];        // touched vertices, flipped rows
    unsigned long long nsegs[4]; // segments of the frontier's long rows
    unsigned long long dd[4];    // change of P
    unsigned long long dmask[4], dent[4];  // upper entries and entries that left
    unsigned long long bar;      // arrivals at the barrier
    // iters .. ent are read back together
    int32_t iters;               // reported iteration count
    int32_t failed;              // a wait at the one-launch loop's barrier ran out
    int32_t live;                // batches: graphs still iterating (from here on kept from one k to the next)
    int32_t diag;                // the matrix has diagonal entries
    unsigned long long ent;      // entries of C_t
    unsigned long long prod;     // P_t (batches: summed over the live graphs)
    unsigned long long mask;     // entries (i, j) of C_t with j >= i
};
struct TriFrontResult {
    int32_t iters, failed, live, diag;
    unsigned long long ent;
};
static_assert(offsetof(TriFrontState, ent) - offsetof(TriFrontState, iters) == offsetof(TriFrontResult, ent),
              "the part of the state that is read back");

struct TriFrontArgs {
    const int32_t* cr;      // row starts (fixed during the loop)
    const int32_t* cc;      // columns, every row as [oriented part | rest]
    const int32_t* ac;      // columns, rows in column order
    const int32_t* row_of;
    const int32_t* crank;   // rank of each entry's column
    const int32_t* rank;    // of each vertex
    const int32_t* ocount;
    const int32_t* dpos;    // position of each row's diagonal entry, -1 if none
    int32_t* oid;           // entry (of cc) -> position of its edge's record
    int32_t* orec;          // the same for the entries in column order (of ac)
    int32_t* sup;           // supports at the records
    uint8_t* state;         // states at the records
    int32_t* deg;           // entries of each row still in C
    int32_t* upc;           // of those, the ones with column >= row
    uint8_t* h;             // upc > 0, as of the iteration's start
    int32_t* H;             // per vertex: entries (i, j) of C with h(i) = 1
    int32_t* rd;            // per vertex: entries its row lost this iteration
    int32_t* rh;            // per vertex: what H lost this iteration
    int32_t* mark;          // per vertex: listed in touched
    int32_t* touched;
    int32_t* flip;
    int32_t* f0;
    int32_t* f1;
    int2* seg;              // segments of long rows: (frontier slot, segment)
    int32_t* efound;        // per frontier slot: triangles its segments found
    int64_t segcap;
    TriFrontState* st;
    unsigned long long* ctr;
    int64_t m;
    int64_t nnz;
    int k;
    // batches of graphs (block-diagonal union; gid == nullptr: one matrix)
    const int32_t* gid;     // graph of each row
    const int32_t* kg;      // per-graph k (nullptr: k for every graph)
    const int32_t* nvert;   // vertices per graph
    int32_t* done_g;        // graph finished (converged, or stopped after n_g iterations)
    int32_t* iters_g;       // reported iteration count per graph
    int32_t* cntg;          // 2 x ngraphs: frontier elements per graph, by iteration parity
    long long* pg;          // P per graph
    int64_t ngraphs;
    // one-launch loop: further buffers (used in turn by the iterations), row
    // lengths of the rows with a diagonal entry
    int32_t *rd1, *rd2, *rh1, *rh2, *touched1, *touched2, *flip1, *flip2;
    int32_t* dcur;
    int2* seg1;
    int64_t segcap1;        // of seg and seg1
};

__device__ __forceinline__ void front_push(int32_t* buf, int32_t* cnt, int32_t x) { buf[atomicAdd(cnt, 1)] = x; }

// k - 2 for the graph of row i
__device__ __forceinline__ int kt_thr(const TriFrontArgs& a, int32_t i) {
    return (a.kg ? a.kg[a.gid[i]] : a.k) - 2;
}

// A frontier element of row i for iteration parity par (batches also count
// it for the row's graph).
__device__ __forceinline__ void front_add(const TriFrontArgs& a, int32_t* buf, int32_t* cnt, int32_t x, int32_t i,
                                          int par) {
    front_push(buf, cnt, x);
    if (a.gid) atomicAdd(a.cntg + par * a.ngraphs + a.gid[i], 1);
}

// Batches: the element's graph finished (a graph stopped by its iteration
// bound keeps its edges; its queued elements are dropped).
__device__ __forceinline__ bool kt_frozen(const TriFrontArgs& a, int32_t i) {
    return a.gid && a.done_g[a.gid[i]];
}

// One support unit less; the edge joins the next frontier when it drops below k - 2.
__device__ __forceinline__ void lower_support(const TriFrontArgs& a, int32_t f, int32_t* fn, int32_t* cn, int par) {
    if (!a.gid) {
        if (atomicSub(a.sup + f, 1) == a.k - 2) front_push(fn, cn, f);
        return;
    }
    const int32_t i = a.row_of[f];
    if (atomicSub(a.sup + f, 1) == kt_thr(a, i)) front_add(a, fn, cn, f, i, par);
}

__device__ __forceinline__ void touch(const TriFrontArgs& a, int32_t x) {
    if (atomicExch(a.mark + x, 1) == 0) front_push(a.touched, &a.st->ntouch, x);
}

__global__ void k_trif_init_rows(TriFrontArgs a) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < a.m; i += (int64_t)gridDim.x * blockDim.x) {
        const int32_t b = a.cr[i], n = a.cr[i + 1] - b;
        const int32_t up = n - lower_bound_i32(a.ac + b, n, (int32_t)i);
        a.deg[i] = n;
        a.upc[i] = up;
        a.h[i] = up > 0;
        a.H[i] = 0;
        a.rd[i] = 0;
        a.rh[i] = 0;
        a.mark[i] = 0;
        if (a.dcur) {
            a.rd1[i] = a.rd2[i] = 0;
            a.rh1[i] = a.rh2[i] = 0;
            a.dcur[i] = n;
        }
    }
}

// The states, every entry's record (the oriented entry of its edge; a diagonal entry is
// its own), for the entries as the loop stores them and in column order, the
// diagonal positions, and H. An oriented entry is its own record, the other
// entry of the edge searches the row ranked below for it, in the short
// oriented part. (A mirror found for both, each by its own search, then a
// pass to make records of them, and H by a warp per row, where a hub's row
// keeps one warp busy: 389 us together at R-MAT 18 and 1,190 us for 512
// nearest-neighbour graphs of 46M entries.)
__global__ void k_trif_records(TriFrontArgs a, WordRanks r, int32_t* __restrict__ dpos) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t threads = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~(int64_t)31; p0 < a.nnz; p0 += threads) {
        const int64_t p = p0 + lane;
        int32_t i = -1;
        bool hj = false;
        if (p < a.nnz) {
            i = a.row_of[p];
            const int32_t j = a.ac[p];
            bool o;
            const int32_t np = part_place(r, p, a.cr[i], a.ocount[i], &o);
            int32_t rec = np;
            if (i == j) {
                dpos[i] = np;
                a.st->diag = 1;
            } else if (!o) {
                const int32_t jb = a.cr[j];
                rec = jb + lower_bound_i32(a.cc + jb, a.ocount[j], i);
            }
            a.orec[p] = rec;
            a.oid[np] = rec;
            a.state[p] = kAlive;
            hj = a.h[j] != 0;
        }
        // entries of each row among the warp's
        const int32_t before = __shfl_up_sync(FULL, i, 1);
        const unsigned heads = __ballot_sync(FULL, lane == 0 || before != i), set = __ballot_sync(FULL, hj);
        if (i >= 0 && (heads >> lane & 1u)) {
            const unsigned later = heads & ~((2u << lane) - 1u);
            const unsigned upto = later ? (1u << (__ffs(later) - 1)) - 1u : FULL;
            const int c = __popc(set & upto & ~((1u << lane) - 1u));
            if (c) atomicAdd(a.H + i, c);
        }
    }
}

// A warp's records of the first frontier, kSeedWords words of 32 entries from
// q0 on (is: bit w for the lane's entry of word w): they take their places
// together, since all places come from one counter (R-MAT 18's 4-truss, half
// of the records in the first frontier: an atomic per word 52 us, per four
// words 30). One matrix: the records are marked at once; batches mark
// theirs in k_trif_mark and count them for their graphs.
constexpr int kSeedWords = 4;
__device__ __forceinline__ void front_first(const TriFrontArgs& a, unsigned is, int64_t q0) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int mine = __popc(is), incl = warp_incl_scan(mine), total = __shfl_sync(FULL, incl, 31);
    if (!total) return;
    int32_t at = 0;
    if (lane == 0) at = atomicAdd(&a.st->cnt[0], total);
    at = __shfl_sync(FULL, at, 0) + incl - mine;
    for (; is; is &= is - 1) {
        const int32_t q = (int32_t)q0 + (__ffs(is) - 1) * 32 + lane;
        a.f0[at++] = q;
        if (a.gid) atomicAdd(a.cntg + a.gid[a.row_of[q]], 1);
        else a.state[q] = kDying;
    }
}

// The diagonal terms of the listed supports, and the first frontier. (The
// states are alive.)
__global__ void k_trif_seed(TriFrontArgs a) {
    const bool diag = a.st->diag != 0;
    const int lane = threadIdx.x & 31;
    const int64_t step = (int64_t)gridDim.x * (blockDim.x >> 5) * kSeedWords * 32;
    for (int64_t q0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kSeedWords * 32; q0 < a.nnz;
         q0 += step) {
        unsigned is = 0;
#pragma unroll
        for (int w = 0; w < kSeedWords; ++w) {
            const int64_t q = q0 + w * 32 + lane;
            if (q >= a.nnz || a.oid[q] != (int32_t)q) continue;
            int32_t s = a.sup[q];
            if (diag) {
                const int32_t i = a.row_of[q], j = a.cc[q];
                if (i == j) {
                    s = a.deg[i];
                } else {
                    s += (a.dpos[i] >= 0) + (a.dpos[j] >= 0);
                    a.sup[q] = s;
                }
            }
            is |= (unsigned)(s < (a.kg ? kt_thr(a, a.row_of[q]) : a.k - 2)) << w;
        }
        front_first(a, is, q0);
    }
}

// A later k of a sweep (one matrix): the edges left by the previous k have
// exact supports in C, so the first frontier of the new k is the live
// records below the new k - 2 (a diagonal record: its row's length).
__global__ void k_trif_reseed(TriFrontArgs a) {
    const bool diag = a.st->diag != 0;
    const int lane = threadIdx.x & 31;
    const int64_t step = (int64_t)gridDim.x * (blockDim.x >> 5) * kSeedWords * 32;
    for (int64_t q0 = (((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5) * kSeedWords * 32; q0 < a.nnz;
         q0 += step) {
        unsigned is = 0;
#pragma unroll
        for (int w = 0; w < kSeedWords; ++w) {
            const int64_t q = q0 + w * 32 + lane;
            if (q >= a.nnz || a.oid[q] != (int32_t)q || a.state[q] != kAlive) continue;
            const int32_t s = diag && a.cc[q] == a.row_of[q] ? a.deg[a.row_of[q]] : a.sup[q];
            is |= (unsigned)(s < a.k - 2) << w;
        }
        front_first(a, is, q0);
    }
}

// P_0, the upper entries and the entries of C_0; one thread per row.
__global__ void k_trif_init_counts(TriFrontArgs a) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t threads = (int64_t)gridDim.x * blockDim.x;
    unsigned long long prod = 0, mask = 0, ent = 0;
    for (int64_t j0 = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) & ~(int64_t)31; j0 < a.m; j0 += threads) {
        const int64_t j = j0 + lane;
        unsigned long long pj = 0;
        if (j < a.m) {
            pj = (unsigned long long)a.deg[j] * (unsigned long long)a.H[j];
            mask += (unsigned long long)a.upc[j];
            ent += (unsigned long long)a.deg[j];
        }
        prod += pj;
        if (a.gid) {
            // most warps lie inside one graph
            const int32_t g = a.gid[min(j, a.m - 1)], g0 = __shfl_sync(FULL, g, 0);
            const bool one = __all_sync(FULL, g == g0);
            if (one) pj = warp_sum<unsigned long long>(pj);
            if (pj && (!one || lane == 0)) atomicAdd(reinterpret_cast<unsigned long long*>(a.pg + g), pj);
        }
    }
    prod = warp_sum<unsigned long long>(prod);
    mask = warp_sum<unsigned long long>(mask);
    ent = warp_sum<unsigned long long>(ent);
    if (lane == 0) {
        if (prod) atomicAdd(&a.st->prod, prod);
        if (mask) atomicAdd(&a.st->mask, mask);
        if (ent) atomicAdd(&a.st->ent, ent);
    }
    // batches: the graphs still to iterate
    if (a.gid)
        for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < a.ngraphs;
             g += (int64_t)gridDim.x * blockDim.x)
            if (!a.done_g[g]) atomicAdd(&a.st->live, 1);
}

// The reference's work for one iteration's support product C_t * C_t (its
// Gustavson products, mask and stored entries), added to the context's
// counters by one thread.
__device__ __forceinline__ void trif_count_iteration(const TriFrontArgs& a) {
    atomicAdd(&a.ctr[GA_CTR_PRODUCTS], a.st->prod);
    atomicAdd(&a.ctr[GA_CTR_MASK_ENTRIES], a.st->mask);
    atomicAdd(&a.ctr[GA_CTR_A_ENTRIES], a.st->ent);
    atomicAdd(&a.ctr[GA_CTR_LAUNCHES], 1ull);
    atomicAdd(&a.ctr[GA_CTR_ROWS], (unsigned long long)a.m);
}

// One matrix, before a k's first iteration (whose frontier the seed marked):
// that iteration's counters. Later iterations are counted by k_trif_delta.
__global__ void k_trif_begin(TriFrontArgs a) {
    if (blockIdx.x == 0 && threadIdx.x == 0) trif_count_iteration(a);
}

// Batches, start of iteration t: the work counters of its support product,
// and the frontier marked.
__global__ void k_trif_mark(const TriFrontArgs* __restrict__ ap) {
    const TriFrontArgs a = *ap;
    const int t = a.st->t;
    const int32_t n = a.st->cnt[t & 1];
    const int32_t* F = (t & 1) ? a.f1 : a.f0;
    if (blockIdx.x == 0 && threadIdx.x == 0) trif_count_iteration(a);
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
        const int32_t q = F[x];
        if (!kt_frozen(a, a.row_of[q])) a.state[q] = kDying;
    }
}

// Rows of at most this many entries are staged in shared memory (columns
// and record positions) before the probes search them.
constexpr int kTrifStage = 256;  // (512: 2 % slower sweep, twice the shared memory)
// An edge whose shorter row has more than kTrifSplit entries is walked in
// segments of kTrifSeg entries by separate warps (k_trif_lower_seg).
constexpr int kTrifSplit = 128;
constexpr int kTrifSeg = 64;
// Grids of the loop's kernels, per SM: the pruning kernels (128 threads)
// and the passes over the frontier (256 threads).
constexpr int kTrifLowerCtas = 8;
constexpr int kTrifPassCtas = 2;

// A frontier edge (u, v) to walk: the shorter row x, the other row y with
// its oriented part [yb, yo) and the rest [yo, ye), y's rank, and the
// triangles the edge is in (its support without the diagonal terms).
struct TrifEdge {
    int32_t q, u, v, xb, xe, yb, yo, ye, ry;
    int target;
};

// The states of the records as an iteration sees them. The captured loop's
// kernels mark them between the iterations.
struct TrifMarked {
    __device__ __forceinline__ uint8_t operator()(uint8_t s) const { return s; }
};

// diag: the matrix has diagonal entries.
template <typename State>
__device__ __forceinline__ TrifEdge trif_edge(const TriFrontArgs& a, int32_t q, int32_t u, int32_t v,
                                              const State& now, bool diag) {
    TrifEdge e;
    e.q = q;
    e.u = u;
    e.v = v;
    e.target = a.sup[q];
    if (diag) {
        const int32_t du = a.dpos[u], dv = a.dpos[v];
        e.target -= (du >= 0 && now(a.state[du]) != kGone) + (dv >= 0 && now(a.state[dv]) != kGone);
    }
    const int32_t ub = a.cr[u], ue = a.cr[u + 1], vb = a.cr[v], ve = a.cr[v + 1];
    const bool xu = ue - ub <= ve - vb;  // walk the shorter row
    e.xb = xu ? ub : vb;
    e.xe = xu ? ue : ve;
    const int32_t y = xu ? v : u;
    e.yb = xu ? vb : ub;
    e.ye = xu ? ve : ue;
    e.yo = e.yb + a.ocount[y];
    e.ry = a.rank[y];
    return e;
}

// Row y of an edge as the lookups see it: columns and record positions from
// yb on, in shared memory (a short row) or in global memory; with shift > 0,
// shared memory holds every 2^shift-th column, which leaves `shift` dependent
// loads of a search in global memory (a hub's row took up to 15).
struct TrifRow {
    const int32_t* col;
    const int32_t* oid;
    const int32_t* fence;  // columns 0, 2^shift, 2 * 2^shift, ...
    int shift;             // 0: none
};

// First position >= sb and < se (one of y's parts, sorted) whose column is at
// least w; se if none.
__device__ __forceinline__ int32_t trif_search(const TrifRow& y, int32_t sb, int32_t se, int32_t w) {
    if (y.shift) {
        // fences inside the part: i0 .. i1 - 1
        const int32_t up = (1 << y.shift) - 1, i0 = (sb + up) >> y.shift, i1 = (se + up) >> y.shift;
        const int32_t k = i0 + lower_bound_i32(y.fence + i0, i1 - i0, w);
        if (k > i0) sb = ((k - 1) << y.shift) + 1;
        if (k < i1) se = k << y.shift;
    }
    return sb + lower_bound_i32(y.col + sb, se - sb, w);
}

// Entry p of row x looked up in row y; loads only, and the independent ones
// first, so that they overlap. A hit is the triangle (u, v, w): f and g are
// the records of its other two edges (u or v, w) and (y, w), with their
// states.
struct TrifHit {
    int32_t f, g, w;
    uint8_t sf, sg;
    bool hit;
};

template <typename State>
__device__ __forceinline__ TrifHit trif_find(const TriFrontArgs& a, const TrifEdge& e, int32_t p, const TrifRow& y,
                                             const State& now) {
    TrifHit h;
    h.hit = false;
    h.g = 0;
    h.sg = kGone;
    const int32_t w = a.cc[p], rank = a.crank[p];
    h.w = w;
    h.f = a.oid[p];
    h.sf = now(a.state[h.f]);
    if (w == e.u || w == e.v) return h;
    // w ranked above y: (y, w) is in y's oriented part
    const bool above = rank > e.ry;
    const int32_t sb = above ? 0 : e.yo - e.yb, se = above ? e.yo - e.yb : e.ye - e.yb;
    const int32_t r = trif_search(y, sb, se, w);
    if (r >= se || y.col[r] != w) return h;
    h.g = y.oid[r];
    h.sg = now(a.state[h.g]);
    h.hit = h.sf != kGone && h.sg != kGone;
    return h;
}

// A hit lowers the supports of the triangle's other two edges, each once
// (the frontier edge with the smallest record position owns a triangle with
// two frontier edges): lower(record, length of the row x or y, w).
template <typename Lower>
__device__ __forceinline__ void trif_apply_hit(const TrifEdge& e, const TrifHit& h, const Lower& lower) {
    if (!h.hit) return;
    if (h.sf == kAlive && (h.sg == kAlive || e.q < h.g)) lower(h.f, e.xe - e.xb, h.w);
    if (h.sg == kAlive && (h.sf == kAlive || e.q < h.f)) lower(h.g, e.ye - e.yb, h.w);
}

// A warp walks entries [p0, p1) of the edge's shorter row, 32 per pass (two
// per lane per pass were slower: the later stop wastes more lookups than the
// overlap gains), stopping once the edge's triangles are found. found: the
// edge's count, shared by the warps that walk its segments (nullptr: this
// warp walks the whole row).
template <typename State, typename Lower>
__device__ __forceinline__ void trif_walk(const TriFrontArgs& a, const TrifEdge& e, int32_t p0, int32_t p1,
                                          const TrifRow& y, int32_t* found, const State& now, const Lower& lower,
                                          unsigned long long& probes, unsigned long long& tris) {
    const int lane = threadIdx.x & 31;
    int mine = 0;
    for (int32_t base = p0; base < p1; base += 32) {
        const int32_t p = base + lane;
        TrifHit h;
        h.hit = false;
        if (p < p1) {
            ++probes;
            h = trif_find(a, e, p, y, now);
            trif_apply_hit(e, h, lower);
        }
        const int hcount = __popc(__ballot_sync(0xffffffffu, h.hit));
        mine += hcount;
        if (lane == 0) tris += (unsigned long long)hcount;
        if (found) {
            if (lane == 0)
                mine = hcount ? atomicAdd(found, hcount) + hcount : *(volatile int32_t*)found;
            mine = __shfl_sync(0xffffffffu, mine, 0);
        }
        if (mine >= e.target) break;
    }
}

// The edge's other row through the warp's 2 * kTrifStage words of shared
// memory: copied there (columns and record positions) when it has at most
// kTrifStage entries, else its fences.
__device__ __forceinline__ TrifRow trif_stage(const TriFrontArgs& a, const TrifEdge& e, int32_t* buf) {
    const int lane = threadIdx.x & 31;
    const int32_t n = e.ye - e.yb;
    TrifRow y;
    __syncwarp();  // the previous edge's lookups are done
    if (n <= kTrifStage) {
        for (int32_t i = lane; i < n; i += 32) {
            buf[i] = a.cc[e.yb + i];
            buf[kTrifStage + i] = a.oid[e.yb + i];
        }
        y.col = buf;
        y.oid = buf + kTrifStage;
        y.shift = 0;
    } else {
        y.shift = 1;
        while (((n - 1) >> y.shift) >= 2 * kTrifStage) ++y.shift;
        for (int32_t i = lane; i <= (n - 1) >> y.shift; i += 32) buf[i] = a.cc[e.yb + (i << y.shift)];
        y.col = a.cc + e.yb;
        y.oid = a.oid + e.yb;
    }
    y.fence = buf;
    __syncwarp();
    return y;
}

// One warp per frontier edge: its triangles in C_t, the supports they lower.
// The warp walks the shorter row x of the edge and looks each entry up in
// the other row y: in y's part that the entry's rank selects, binary-searched
// in shared memory when y has at most kTrifStage entries (its columns and
// record positions copied there first, coalesced), else in global memory.
// A row x longer than kTrifSplit is listed as segments for
// k_trif_lower_seg instead (while the segment list has room).
__global__ void __launch_bounds__(128, 8) k_trif_lower(const TriFrontArgs* __restrict__ ap) {
    __shared__ int32_t s_row[4][2 * kTrifStage];
    const TriFrontArgs a = *ap;
    const int lane = threadIdx.x & 31;
    const int t = a.st->t;
    const int32_t n = a.st->cnt[t & 1];
    const int32_t* F = (t & 1) ? a.f1 : a.f0;
    int32_t* fn = (t & 1) ? a.f0 : a.f1;
    int32_t* cn = &a.st->cnt[(t + 1) & 1];
    const int np = (t + 1) & 1;
    auto lower = [&](int32_t f, int32_t, int32_t) { lower_support(a, f, fn, cn, np); };
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    unsigned long long probes = 0, tris = 0, edges = 0;
    for (int64_t x = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < n; x += warps) {
        const int32_t q = F[x];
        const int32_t u = a.row_of[q], v = a.cc[q];
        if (kt_frozen(a, u)) continue;
        if (lane == 0) ++edges;
        if (u == v) {
            // a diagonal entry leaves: every other edge of its row loses 1
            for (int32_t p = a.cr[u] + lane; p < a.cr[u + 1]; p += 32) {
                if (a.cc[p] == u) continue;
                const int32_t f = a.oid[p];
                if (a.state[f] == kAlive) lower_support(a, f, fn, cn, np);
            }
            continue;
        }
        const TrifEdge e = trif_edge(a, q, u, v, TrifMarked(), true);
        if (e.target <= 0) continue;
        if (e.xe - e.xb > kTrifSplit) {
            // segments for k_trif_lower_seg: (frontier slot, segment)
            const int nseg = (e.xe - e.xb + kTrifSeg - 1) / kTrifSeg;
            int base = 0;
            if (lane == 0) base = atomicAdd(&a.st->nseg, nseg);
            base = __shfl_sync(0xffffffffu, base, 0);
            if ((int64_t)base + nseg <= a.segcap) {
                if (lane == 0) a.efound[x] = 0;
                for (int j = lane; j < nseg; j += 32) a.seg[base + j] = make_int2((int32_t)x, j);
                continue;
            }
            // no room: holes in the list are marked, the warp walks the row
            for (int64_t j = base + lane; j < a.segcap && j < (int64_t)base + nseg; j += 32)
                a.seg[j] = make_int2(-1, 0);
        }
        trif_walk(a, e, e.xb, e.xe, trif_stage(a, e, s_row[threadIdx.x >> 5]), nullptr, TrifMarked(), lower, probes, tris);
    }
    probes = warp_sum<unsigned long long>(probes);
    if (lane == 0) {
        if (edges) atomicAdd(&a.ctr[GA_CTR_FRONT_EDGES], edges);
        if (probes) atomicAdd(&a.ctr[GA_CTR_FRONT_PROBES], probes);
        if (tris) atomicAdd(&a.ctr[GA_CTR_FRONT_TRIANGLES], tris);
    }
}

// The segments k_trif_lower listed, one warp each: kTrifSeg entries of a
// long row x looked up in y in global memory. The edge's triangles found so
// far are counted in efound (per frontier slot); a segment stops once they
// reach the edge's total.
__global__ void __launch_bounds__(128, 8) k_trif_lower_seg(const TriFrontArgs* __restrict__ ap) {
    const TriFrontArgs a = *ap;
    const int lane = threadIdx.x & 31;
    const int t = a.st->t;
    const int32_t* F = (t & 1) ? a.f1 : a.f0;
    int32_t* fn = (t & 1) ? a.f0 : a.f1;
    int32_t* cn = &a.st->cnt[(t + 1) & 1];
    const int np = (t + 1) & 1;
    auto lower = [&](int32_t f, int32_t, int32_t) { lower_support(a, f, fn, cn, np); };
    const int64_t ns = min((int64_t)a.st->nseg, a.segcap);
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    unsigned long long probes = 0, tris = 0;
    for (int64_t sx = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; sx < ns; sx += warps) {
        const int2 sg = a.seg[sx];
        if (sg.x < 0) continue;
        const int32_t q = F[sg.x];
        const TrifEdge e = trif_edge(a, q, a.row_of[q], a.cc[q], TrifMarked(), true);
        if (*(volatile int32_t*)(a.efound + sg.x) >= e.target) continue;
        const int32_t s0 = e.xb + sg.y * kTrifSeg, s1 = min(e.xe, s0 + kTrifSeg);
        const TrifRow y{a.cc + e.yb, a.oid + e.yb, nullptr, 0};
        trif_walk(a, e, s0, s1, y, a.efound + sg.x, TrifMarked(), lower, probes, tris);
    }
    probes = warp_sum<unsigned long long>(probes);
    if (lane == 0) {
        if (probes) atomicAdd(&a.ctr[GA_CTR_FRONT_PROBES], probes);
        if (tris) atomicAdd(&a.ctr[GA_CTR_FRONT_TRIANGLES], tris);
    }
}

// The frontier's edges leave C_t: rows shorten (diagonal entries whose row
// length drops below k - 2 join the next frontier), the terms of P at their
// endpoints change, rows that lose their last upper entry are listed.
__global__ void k_trif_apply(const TriFrontArgs* __restrict__ ap) {
    const TriFrontArgs a = *ap;
    const int t = a.st->t;
    const int32_t n = a.st->cnt[t & 1];
    const int32_t* F = (t & 1) ? a.f1 : a.f0;
    int32_t* fn = (t & 1) ? a.f0 : a.f1;
    int32_t* cn = &a.st->cnt[(t + 1) & 1];
    const int np = (t + 1) & 1;
    unsigned long long mask = 0, ent = 0;
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
        const int32_t q = F[x];
        const int32_t u = a.row_of[q], v = a.cc[q];
        if (kt_frozen(a, u)) continue;
        a.state[q] = kGone;
        ++mask;
        // deg and H keep their values from the iteration's start; the losses
        // are counted in rd and rh and applied by k_trif_delta
        if (u == v) {
            ++ent;
            atomicAdd(a.rd + u, 1);
            atomicAdd(a.rh + u, 1);  // h(u) = 1 while its diagonal entry is there
            touch(a, u);
            if (atomicSub(a.upc + u, 1) == 1) front_push(a.flip, &a.st->nflip, u);
            continue;
        }
        ent += 2;
        // the row lengths before this entry left
        const int32_t ou = a.deg[u] - atomicAdd(a.rd + u, 1), ov = a.deg[v] - atomicAdd(a.rd + v, 1);
        if (a.h[u]) atomicAdd(a.rh + v, 1);
        if (a.h[v]) atomicAdd(a.rh + u, 1);
        touch(a, u);
        touch(a, v);
        const int32_t lo = min(u, v);
        if (atomicSub(a.upc + lo, 1) == 1) front_push(a.flip, &a.st->nflip, lo);
        // a diagonal entry's support is its row's length
        if (ou == kt_thr(a, u)) {
            const int32_t d = a.dpos[u];
            if (d >= 0 && a.state[d] == kAlive) front_add(a, fn, cn, d, u, np);
        }
        if (ov == kt_thr(a, v)) {
            const int32_t d = a.dpos[v];
            if (d >= 0 && a.state[d] == kAlive) front_add(a, fn, cn, d, v, np);
        }
    }
    mask = warp_sum<unsigned long long>(mask);
    ent = warp_sum<unsigned long long>(ent);
    if ((threadIdx.x & 31) == 0 && mask) {
        atomicAdd(&a.st->mask, (unsigned long long)(-(long long)mask));
        atomicAdd(&a.st->ent, (unsigned long long)(-(long long)ent));
    }
}

// Rows that lost their last upper entry: h drops to 0, so every remaining
// neighbour's H loses 1. One warp per row.
// H(j) loses 1 here directly, and P loses deg(j) (the row length at the
// iteration's start): k_trif_delta's term for a touched j, computed from
// this H, then misses exactly that; a j that nothing else touched changes
// by exactly that. So the flipped rows' neighbours are neither touched nor
// counted in rh.
__global__ void k_trif_flip(const TriFrontArgs* __restrict__ ap) {
    const TriFrontArgs a = *ap;
    const int lane = threadIdx.x & 31;
    const int32_t n = a.st->nflip;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    long long d = 0;  // this lane's part of the change of P
    for (int64_t x = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; x < n; x += warps) {
        const int32_t i = a.flip[x];
        if (lane == 0) a.h[i] = 0;
        long long di = 0;
        for (int32_t p = a.cr[i] + lane; p < a.cr[i + 1]; p += 32) {
            if (a.state[a.oid[p]] == kGone) continue;
            const int32_t j = a.cc[p];
            atomicSub(a.H + j, 1);
            di -= a.deg[j];
        }
        if (a.gid) {
            // the neighbours of row i are in i's graph
            const long long gi = warp_sum<long long>(di);
            if (lane == 0 && gi) atomicAdd(reinterpret_cast<unsigned long long*>(a.pg + a.gid[i]), (unsigned long long)gi);
        }
        d += di;
    }
    d = warp_sum<long long>(d);
    if (lane == 0 && d) atomicAdd(&a.st->prod, (unsigned long long)d);
}

// P_{t+1} = P_t + the change of deg(j) H(j) at every touched vertex (for a
// batch also per graph). For one matrix, the last block to finish ends the
// iteration (stop when F_t was empty, or after m iterations) and tells the
// loop whether to go on; batches end it in k_trif_graphs.
__global__ void __launch_bounds__(256) k_trif_delta(const TriFrontArgs* __restrict__ ap, LoopCtl ctl) {
    const TriFrontArgs a = *ap;
    __shared__ long long part[8];
    __shared__ bool last;
    const int32_t n = a.st->ntouch;
    if (!a.gid) {
        // one matrix: the next frontier is complete, so its edges are marked
        // here instead of by a marking kernel at the next iteration's start
        const int t = a.st->t;
        const int32_t nn = a.st->cnt[(t + 1) & 1];
        const int32_t* Fn = (t & 1) ? a.f0 : a.f1;
        for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < nn; x += (int64_t)gridDim.x * blockDim.x)
            a.state[Fn[x]] = kDying;
    }
    long long d = 0;
    for (int64_t x = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; x < n; x += (int64_t)gridDim.x * blockDim.x) {
        const int32_t j = a.touched[x];
        const long long od = a.deg[j], oh = a.H[j];
        const long long nd = od - a.rd[j], nh = oh - a.rh[j];
        const long long dj = nd * nh - od * oh;
        d += dj;
        if (a.gid && dj) atomicAdd(reinterpret_cast<unsigned long long*>(a.pg + a.gid[j]), (unsigned long long)dj);
        a.deg[j] = (int32_t)nd;
        a.H[j] = (int32_t)nh;
        a.rd[j] = 0;
        a.rh[j] = 0;
        a.mark[j] = 0;
    }
    d = warp_sum<long long>(d);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = d;
    __syncthreads();
    if (threadIdx.x == 0) {
        long long s = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) s += part[w];
        if (s) atomicAdd(&a.st->prod, (unsigned long long)s);
        __threadfence();
        last = atomicAdd(&a.st->blocks_done, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    __threadfence();
    TriFrontState* st = a.st;
    st->blocks_done = 0;
    st->ntouch = 0;
    st->nflip = 0;
    st->nseg = 0;
    if (a.gid) return;
    const int t = st->t;
    if (st->cnt[t & 1] == 0) {
        st->iters = t + 1;
        st->done = 1;
    } else {
        st->cnt[t & 1] = 0;
        st->t = t + 1;
        if ((int64_t)(t + 1) >= a.m) {
            st->iters = 0;
            st->done = 1;
        }
    }
    if (!st->done) trif_count_iteration(a);
    loop_continue(ctl, st->done == 0);
}

// ------------------------------------------------- the loop in one launch
// One matrix, device loops: the iterations of a run(k) inside one cooperative
// launch, one CTA per SM, one grid barrier per iteration. As five kernels per
// iteration of a captured loop, an iteration with a few hundred frontier edges
// took 35 us and its loop node 8 more, most of it launches, their tails and
// chains of dependent loads; here it takes 13 to 16 us, of which the barrier is
// 2.3 and the rest the longest chain (queue entry, edge, rows, staging, lookup,
// support, queue). R-MAT 18 sweep, 1,412 iterations: 33.5 ms of 54 in the loop,
// 56 of 86 before (two barriers per iteration, the parts of an iteration one
// after the other: 47.5 of 74). Frontiers above 4,096 edges (167 iterations, 12
// ms) are bound by how many of these chains 32 warps per SM have in flight.
//
// What an iteration needs from the one before is only its frontier and the
// supports, so stage s runs
//   A(s)    the frontier's triangles lower the supports (k_trif_lower),
//           queueing and marking the edges that cross k - 2 for s + 1
//   B(s-1)  the counts of what left in iteration s - 1 (k_trif_apply)
//   C(s-2)  the rows that lost their last upper entry in iteration s - 2
//           lower their neighbours' H (k_trif_flip)
//   D(s-3)  the vertices touched in iteration s - 3 get their new row lengths
//           and H, and P its change (k_trif_delta); its edges become kGone
// side by side, and three stages after the last iteration settle the rest.
// * A queued edge's state is the code 3 + (its iteration mod 5) until D: in
//   stage s the code of s + 1 means alive, of s dying, of s - 1 .. s - 3 gone,
//   and the code of s - 4 (that of s + 1) is no longer in use.
// * Every edge leaves once, so all frontiers of a run share one list, one
//   after the other; iteration t's counters are slot t mod 4 (reset by the
//   settling thread when nothing reads them), its buffers t mod 3, and a row
//   flipped in iteration t has h = 2 + t mod 3 until C.
// * A diagonal entry joins the next frontier when its row becomes too short,
//   which B finds: with diagonal entries B(s) runs in stage s, behind a
//   barrier of its own.
// * A long row is cut into segments when its edge is queued; while the
//   frontier is small, so that most warps are idle, from 33 entries on.
constexpr int kTrifLoopThreads = 1024;
constexpr int kTrifLoopWarps = kTrifLoopThreads / 32;
constexpr size_t kTrifLoopSmem = (size_t)kTrifLoopWarps * kTrifStage * 2 * sizeof(int32_t);
constexpr int kTrifFine = 8;  // warps of the grid per frontier edge from which rows are cut finely
constexpr long long kTrifWaitCycles = 20000000000ll;  // about ten seconds at 2 GHz

// All CTAs of the launch (cooperative: they are resident together) have
// arrived `round` times. False when a wait ran out, here or elsewhere.
__device__ __forceinline__ bool trif_barrier(TriFrontState* st, unsigned long long round) {
    __shared__ bool s_ok;
    __syncthreads();
    if (threadIdx.x == 0) {
        __threadfence();
        const unsigned long long all = round * gridDim.x;
        if (atomicAdd(&st->bar, 1ull) + 1ull < all) {
            const long long t0 = clock64();
            while (*(volatile unsigned long long*)&st->bar < all) {
                if (*(volatile int32_t*)&st->failed) break;
                if (clock64() - t0 > kTrifWaitCycles) {
                    atomicExch(&st->failed, 1);
                    break;
                }
            }
        }
        __threadfence();
        s_ok = *(volatile int32_t*)&st->failed == 0;
    }
    __syncthreads();
    return s_ok;
}

__device__ __forceinline__ uint8_t trif_code(int t) { return (uint8_t)(3 + t % 5); }

// The states in stage s.
struct TrifCoded {
    uint8_t next, dying;
    __device__ __forceinline__ explicit TrifCoded(int s) : next(trif_code(s + 1)), dying(trif_code(s)) {}
    __device__ __forceinline__ uint8_t operator()(uint8_t v) const {
        return v == kAlive || v == next ? kAlive : v == dying ? kDying : kGone;
    }
};

// Segments of the shorter row (len entries) of the edge at place x of the
// frontier list; efound says whether they were listed.
__device__ __forceinline__ void trif_cut(const TriFrontArgs& a, int32_t x, int32_t len, bool fine, int2* seg,
                                         unsigned long long* nsegs) {
    int32_t listed = -1;
    if (len > (fine ? 32 : kTrifSplit)) {
        const int per = fine ? 32 : kTrifSeg, n = (len + per - 1) / per;
        const int64_t base = (int64_t)atomicAdd(nsegs, (unsigned long long)n);
        if (base + n <= a.segcap1) listed = 0;
        for (int64_t j = 0; j < n && base + j < a.segcap1; ++j)
            seg[base + j] = make_int2(listed < 0 ? -1 : x, (int32_t)(2 * j) | (fine ? 1 : 0));
    }
    a.efound[x] = listed;
}

__global__ void __launch_bounds__(kTrifLoopThreads, 1) k_trif_loop(const __grid_constant__ TriFrontArgs a) {
    extern __shared__ int32_t s_rows[];
    TriFrontState* st = a.st;
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int32_t* buf = s_rows + (size_t)wid * 2 * kTrifStage;
    // warps of one CTA lie apart, so that few items spread over the SMs
    const int64_t warp = (int64_t)wid * gridDim.x + blockIdx.x, warps = (int64_t)gridDim.x * kTrifLoopWarps;
    const int64_t thread = warp * 32 + lane, threads = warps * 32;
    // each part of a stage starts at another quarter of the warps: with few
    // items, the parts run on different warps instead of one after the other
    auto quarter = [&](int q) {
        const int64_t w = warp - q * (warps / 4);
        return w < 0 ? w + warps : w;
    };
    const int64_t warp_b = quarter(1), warp_c = quarter(2), thread_d = quarter(3) * 32 + lane;
    // the thread that keeps the totals: of the warp that gets work last
    const bool settles = thread == threads - 32;
    const bool diag = st->diag != 0;
    const int thr = a.k - 2;
    int32_t* const F = a.f0;
    unsigned long long round = 0, probes = 0, tris = 0, edges = 0;

    // P_it (its change by iteration it - 1 is known), the counters of
    // iteration `it` when it counts, and what left in it. One thread.
    auto settle = [&](int it, bool count) {
        if (it > 0) {
            st->prod += *(volatile unsigned long long*)&st->dd[(it - 1) & 3];
            st->dd[(it - 1) & 3] = 0;
        }
        if (count) trif_count_iteration(a);
        st->mask -= *(volatile unsigned long long*)&st->dmask[it & 3];
        st->ent -= *(volatile unsigned long long*)&st->dent[it & 3];
        st->dmask[it & 3] = 0;
        st->dent[it & 3] = 0;
    };
    // Vertices x (lanes with `is`) newly touched in iteration `it`, listed.
    auto list_touched = [&](int it, bool is, int32_t x) {
        const unsigned b = __ballot_sync(FULL, is);
        if (b == 0u) return;
        int32_t at = 0;
        if (lane == 0) at = atomicAdd(&st->nt[it & 3], __popc(b));
        at = __shfl_sync(FULL, at, 0);
        const int r = it % 3;
        int32_t* list = r == 0 ? a.touched : r == 1 ? a.touched1 : a.touched2;
        if (is) list[at + __popc(b & ((1u << lane) - 1u))] = x;
    };

    // Queueing for iteration it + 1 from stage `it`: record f, whose edge's
    // shorter row has len entries (0: a diagonal entry).
    auto queue = [&](int it, int64_t next_at, bool fine, int32_t f, int32_t len) {
        const int32_t x = (int32_t)next_at + atomicAdd(&st->nfront[(it + 1) & 3], 1);
        F[x] = f;
        a.state[f] = trif_code(it + 1);
        trif_cut(a, x, len, fine, it & 1 ? a.seg : a.seg1, &st->nsegs[(it + 1) & 3]);
    };

    // A(s): items [0, n) the frontier, then its segments
    auto lower_stage = [&](int s, int64_t at, int64_t n, int64_t ns, bool fine) {
        const TrifCoded now(s);
        const int64_t next_at = at + n;
        const int2* seg = s & 1 ? a.seg1 : a.seg;
        auto lower = [&](int32_t f, int32_t len, int32_t w) {
            if (atomicSub(a.sup + f, 1) == thr) queue(s, next_at, fine, f, min(len, a.cr[w + 1] - a.cr[w]));
        };
        for (int64_t x0 = warp; x0 < n + ns; x0 += warps * 32) {
            // the warp's next 32 items, one per lane: their chains of loads
            // overlap
            const int64_t x = x0 + (int64_t)lane * warps;
            TrifEdge e = {};
            int32_t slot = -1, p0 = 0, p1 = 0;
            bool todo = false;
            if (x < n) {
                const int32_t q = F[at + x];
                const int32_t cut = a.efound[at + x];
                const int32_t u = a.row_of[q], v = a.cc[q];
                ++edges;
                if (u == v) {
                    e.u = e.v = u;
                    todo = true;
                } else if (cut < 0) {
                    e = trif_edge(a, q, u, v, now, diag);
                    p0 = e.xb;
                    p1 = e.xe;
                    todo = e.target > 0;
                }
            } else if (x < n + ns) {
                const int2 sg = seg[x - n];
                if (sg.x >= 0) {
                    slot = sg.x;
                    const int32_t q = F[slot], per = sg.y & 1 ? 32 : kTrifSeg;
                    e = trif_edge(a, q, a.row_of[q], a.cc[q], now, diag);
                    p0 = e.xb + (sg.y >> 1) * per;
                    p1 = min(e.xe, p0 + per);
                    todo = *(volatile int32_t*)(a.efound + slot) < e.target;
                }
            }
            for (unsigned set = __ballot_sync(FULL, todo); set; set &= set - 1) {
                const int l = __ffs(set) - 1;
                TrifEdge f;
                f.u = __shfl_sync(FULL, e.u, l);
                f.v = __shfl_sync(FULL, e.v, l);
                if (f.u == f.v) {  // a diagonal entry leaves: every other edge of its row loses 1
                    for (int32_t p = a.cr[f.u] + lane; p < a.cr[f.u + 1]; p += 32) {
                        const int32_t w = a.cc[p];
                        if (w == f.u) continue;
                        const int32_t r = a.oid[p];
                        if (now(a.state[r]) == kAlive) lower(r, a.cr[f.u + 1] - a.cr[f.u], w);
                    }
                    __syncwarp();
                    continue;
                }
                f.q = __shfl_sync(FULL, e.q, l);
                f.xb = __shfl_sync(FULL, e.xb, l);
                f.xe = __shfl_sync(FULL, e.xe, l);
                f.yb = __shfl_sync(FULL, e.yb, l);
                f.yo = __shfl_sync(FULL, e.yo, l);
                f.ye = __shfl_sync(FULL, e.ye, l);
                f.ry = __shfl_sync(FULL, e.ry, l);
                f.target = __shfl_sync(FULL, e.target, l);
                const int32_t b = __shfl_sync(FULL, p0, l), c = __shfl_sync(FULL, p1, l);
                const int32_t sl = __shfl_sync(FULL, slot, l);
                trif_walk(a, f, b, c, trif_stage(a, f, buf), sl < 0 ? nullptr : a.efound + sl, now, lower, probes, tris);
            }
        }
    };
    // B(it)
    auto leave_stage = [&](int it, int64_t at, int64_t n, int64_t next_at) {
        const int r = it % 3, bit = r;
        int32_t* rd = r == 0 ? a.rd : r == 1 ? a.rd1 : a.rd2;
        int32_t* rh = r == 0 ? a.rh : r == 1 ? a.rh1 : a.rh2;
        int32_t* flip = r == 0 ? a.flip : r == 1 ? a.flip1 : a.flip2;
        const uint8_t flipping = (uint8_t)(2 + r);
        unsigned long long mask = 0, ent = 0;
        for (int64_t x0 = warp_b * 32; x0 < n; x0 += threads) {  // whole warps: they reserve places together
            int32_t u = -1, v = -1, lo = 0, du = -1, dv = -1;
            bool tu = false, tv = false, fl = false;  // newly touched, flipped
            if (x0 + lane < n) {
                const int32_t q = F[at + x0 + lane];
                u = a.row_of[q];
                v = a.cc[q];
                ++mask;
                lo = min(u, v);
                // what is read or returned does not wait for one another
                const uint8_t su = a.h[u], sv = a.h[v];
                if (diag && u != v) {
                    du = a.dpos[u];
                    dv = a.dpos[v];
                }
                const int32_t mu = atomicOr(a.mark + u, 1 << bit);
                const int32_t mv = u == v ? -1 : atomicOr(a.mark + v, 1 << bit);
                const int32_t up = atomicSub(a.upc + lo, 1);
                atomicAdd(rd + u, 1);
                if (u != v) atomicAdd(rd + v, 1);
                // h as of the iteration's start: 1, or flipped in it
                if (u == v || su == 1 || su == flipping) atomicAdd(rh + v, 1);
                if (u != v && (sv == 1 || sv == flipping)) atomicAdd(rh + u, 1);
                tu = !(mu >> bit & 1);
                tv = !(mv >> bit & 1);
                fl = up == 1;
                ent += u == v ? 1 : 2;
            }
            list_touched(it, tu, u);
            list_touched(it, tv, v);
            const unsigned bf = __ballot_sync(FULL, fl);
            if (bf) {
                int32_t af = 0;
                if (lane == 0) af = atomicAdd(&st->nf[it & 3], __popc(bf));
                af = __shfl_sync(FULL, af, 0);
                if (fl) {
                    flip[af + __popc(bf & ((1u << lane) - 1u))] = lo;
                    a.h[lo] = flipping;
                }
            }
            // a row that lost an entry: its diagonal entry may become too short
            if (du >= 0 && atomicSub(a.dcur + u, 1) == thr && a.state[du] == kAlive) queue(it, next_at, false, du, 0);
            if (dv >= 0 && atomicSub(a.dcur + v, 1) == thr && a.state[dv] == kAlive) queue(it, next_at, false, dv, 0);
            __syncwarp();
        }
        mask = warp_sum<unsigned long long>(mask);
        ent = warp_sum<unsigned long long>(ent);
        if (lane == 0 && mask) {
            atomicAdd(&st->dmask[it & 3], mask);
            atomicAdd(&st->dent[it & 3], ent);
        }
    };
    // C(it), in stage it + 2: the entries present after iteration `it`
    auto flip_stage = [&](int it) {
        const int32_t n = *(volatile int32_t*)&st->nf[it & 3];
        const int r = it % 3;
        const int32_t* flip = r == 0 ? a.flip : r == 1 ? a.flip1 : a.flip2;
        int32_t* rh = r == 0 ? a.rh : r == 1 ? a.rh1 : a.rh2;
        const uint8_t c1 = trif_code(it + 1), c2 = trif_code(it + 2), c3 = trif_code(it + 3);
        for (int64_t x = warp_c; x < n; x += warps) {
            const int32_t i = flip[x];
            if (lane == 0) a.h[i] = 0;
            const int32_t e = a.cr[i + 1];
            for (int32_t b = a.cr[i]; b < e; b += 32) {
                int32_t j = 0;
                bool is = false;
                if (b + lane < e) {
                    j = a.cc[b + lane];
                    const uint8_t v = a.state[a.oid[b + lane]];
                    if (v == kAlive || v == c1 || v == c2 || v == c3) {
                        atomicAdd(rh + j, 1);
                        is = !(atomicOr(a.mark + j, 1 << r) >> r & 1);
                    }
                }
                list_touched(it, is, j);
            }
        }
    };
    // D(it), in stage it + 3
    auto delta_stage = [&](int it, int64_t at, int64_t nleft) {
        for (int64_t x = thread_d; x < nleft; x += threads) a.state[F[at + x]] = kGone;
        const int32_t n = *(volatile int32_t*)&st->nt[it & 3];
        const int r = it % 3;
        const int32_t* list = r == 0 ? a.touched : r == 1 ? a.touched1 : a.touched2;
        int32_t* rd = r == 0 ? a.rd : r == 1 ? a.rd1 : a.rd2;
        int32_t* rh = r == 0 ? a.rh : r == 1 ? a.rh1 : a.rh2;
        long long d = 0;
        for (int64_t x = thread_d; x < n; x += threads) {
            const int32_t j = list[x];
            const long long od = a.deg[j], oh = a.H[j];
            const long long nd = od - rd[j], nh = oh - rh[j];
            d += nd * nh - od * oh;
            a.deg[j] = (int32_t)nd;
            a.H[j] = (int32_t)nh;
            rd[j] = 0;
            rh[j] = 0;
            atomicAnd(a.mark + j, ~(1 << r));
        }
        d = warp_sum<long long>(d);
        if (lane == 0 && d) atomicAdd(&st->dd[it & 3], (unsigned long long)d);
    };

    // the first frontier: its edges get their code and are cut
    const int64_t n0 = st->cnt[0];
    bool fine = n0 * kTrifFine < warps;
    for (int64_t x = thread; x < n0; x += threads) {
        const int32_t q = F[x], u = a.row_of[q], v = a.cc[q];
        a.state[q] = trif_code(0);
        trif_cut(a, (int32_t)x, u == v ? 0 : min(a.cr[u + 1] - a.cr[u], a.cr[v + 1] - a.cr[v]), fine, a.seg,
                 &st->nsegs[0]);
    }
    bool ok = trif_barrier(st, ++round);
    int64_t n = n0, at = 0;          // this iteration's frontier
    int64_t n1 = 0, n2 = 0, n3 = 0;  // those of the three before
    int last = -1;                   // last iteration with a frontier; -1: not known yet
    int64_t nleft = 0, left_at = 0;  // queued when the bound stopped the loop
    bool ended = false, bound = false;
    for (int s = 0; ok; ++s) {
        if (!ended) {
            if (s > 0) n = *(volatile int32_t*)&st->nfront[s & 3];
            if (n == 0) {
                ended = true;
                last = s - 1;
            }
        } else {
            n = 0;
        }
        if (ended && s > last + 3) break;
        if (ended && last < 0) break;
        const int64_t ns = n ? min((int64_t)*(volatile unsigned long long*)&st->nsegs[s & 3], a.segcap1) : 0;
        fine = n * kTrifFine < warps;
        if (settles) {
            if (s >= 3) settle(s - 3, s - 3 <= last || !ended);
            st->nfront[(s + 2) & 3] = 0;
            st->nsegs[(s + 2) & 3] = 0;
            st->nt[s & 3] = 0;
            st->nf[s & 3] = 0;
        }
        if (n) lower_stage(s, at, n, ns, fine);
        if (n1 && !diag) leave_stage(s - 1, at - n1, n1, 0);
        if (n2) flip_stage(s - 2);
        if (n3) delta_stage(s - 3, at - n1 - n2 - n3, n3);
        if (!(ok = trif_barrier(st, ++round))) break;
        if (n && diag) {
            leave_stage(s, at, n, at + n);
            if (!(ok = trif_barrier(st, ++round))) break;
        }
        at += n;
        n3 = n2;
        n2 = n1;
        n1 = n;
        // the reference's bound: m iterations
        if (!ended && (int64_t)(s + 1) >= a.m) {
            ended = bound = true;
            last = s;
            nleft = *(volatile int32_t*)&st->nfront[(s + 1) & 3];
            left_at = at;
        }
    }
    // (present in C while they had their code)
    for (int64_t x = thread; x < nleft; x += threads) a.state[F[left_at + x]] = kDying;
    if (ok && settles) {
        // the iterations not settled yet (the last one that ran is `last`
        // when the bound stopped the loop, else the empty one after it)
        const int end = bound ? last : last + 1;
        for (int it = last < 0 ? 0 : last + 1; it <= last + 1; ++it) settle(it, it <= end);
        st->iters = bound ? 0 : end + 1;
        st->t = end;
        st->done = 1;
    }
    probes = warp_sum<unsigned long long>(probes);
    edges = warp_sum<unsigned long long>(edges);
    if (lane == 0) {
        if (edges) atomicAdd(&a.ctr[GA_CTR_FRONT_EDGES], edges);
        if (probes) atomicAdd(&a.ctr[GA_CTR_FRONT_PROBES], probes);
        if (tris) atomicAdd(&a.ctr[GA_CTR_FRONT_TRIANGLES], tris);
    }
}

// Batches, end of iteration t, one thread per graph: a live graph without
// frontier elements in this iteration has converged (iteration count t + 1),
// one that reached its bound stops with count 0 (n_g iterations, as the
// reference's loop); both leave the live set and their P leaves the work
// total. The last block ends the iteration; the loop goes on while a graph
// is live.
__global__ void __launch_bounds__(256) k_trif_graphs(const TriFrontArgs* __restrict__ ap, LoopCtl ctl) {
    const TriFrontArgs a = *ap;
    __shared__ long long part[8];
    __shared__ int lpart[8];
    __shared__ bool last;
    const int t = a.st->t;
    int32_t* cnt = a.cntg + (t & 1) * a.ngraphs;
    long long dp = 0;
    int dl = 0;
    for (int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; g < a.ngraphs;
         g += (int64_t)gridDim.x * blockDim.x) {
        const int32_t c = cnt[g];
        cnt[g] = 0;
        if (a.done_g[g]) continue;
        if (c == 0 || (int64_t)(t + 1) >= a.nvert[g]) {
            a.iters_g[g] = c == 0 ? t + 1 : 0;
            a.done_g[g] = 1;
            dp -= a.pg[g];
            ++dl;
        }
    }
    dp = warp_sum<long long>(dp);
    dl = warp_sum<int>(dl);
    if ((threadIdx.x & 31) == 0) {
        part[threadIdx.x >> 5] = dp;
        lpart[threadIdx.x >> 5] = dl;
    }
    __syncthreads();
    if (threadIdx.x == 0) {
        long long s = 0;
        int l = 0;
        for (int w = 0; w < (int)(blockDim.x >> 5); ++w) {
            s += part[w];
            l += lpart[w];
        }
        if (s) atomicAdd(&a.st->prod, (unsigned long long)s);
        if (l) atomicSub(&a.st->live, l);
        __threadfence();
        last = atomicAdd(&a.st->blocks_done_g, 1u) == gridDim.x - 1;
    }
    __syncthreads();
    if (!last || threadIdx.x != 0) return;
    __threadfence();
    TriFrontState* st = a.st;
    st->blocks_done_g = 0;
    st->cnt[t & 1] = 0;
    st->t = t + 1;
    if (st->live <= 0) st->done = 1;
    loop_continue(ctl, st->done == 0);
}

// Keep flags of the entries in column order. One warp per word.
__global__ void k_trif_keep(TriFrontArgs a, WordRanks r) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5), words = a.nnz / 32 + 1;
    for (int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; w < words; w += warps) {
        const int64_t p = w * 32 + lane;
        const unsigned b = __ballot_sync(0xffffffffu, p < a.nnz && a.state[a.orec[p]] != kGone);
        if (lane == 0) {
            r.bits[w] = b;
            r.pre[w] = __popc(b);
        }
    }
}

// After the scan: the kept entries' columns, ones, and the new row starts.
// (Kept entries in the loop's order, each placed by a search of its row's
// other part, with an int per entry as flag and position: flags, scan and
// this 145 us at R-MAT 18.)
__global__ void k_trif_out(TriFrontArgs a, WordRanks r, int32_t* __restrict__ col, int32_t* __restrict__ val,
                           int32_t* __restrict__ rst) {
    const int64_t stride = (int64_t)gridDim.x * blockDim.x;
    for (int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; p < a.nnz || p <= a.m; p += stride) {
        if (p <= a.m) rst[p] = word_rank(r, a.cr[p]);
        if (p < a.nnz && word_flag(r, p)) {
            const int32_t d = word_rank(r, p);
            col[d] = a.ac[p];
            val[d] = 1;
        }
    }
}

}  // namespace

// One CTA of the one-launch loop fits every SM of the context's device.
static bool trif_loop_fits(ga_ctx ctx) {
    static std::mutex mu;
    static std::map<int, bool> known;  // per device
    std::lock_guard<std::mutex> lock(mu);
    auto it = known.find(ctx->device);
    if (it != known.end()) return it->second;
    int coop = 0, per_sm = 0;
    const bool ok =
        cudaDeviceGetAttribute(&coop, cudaDevAttrCooperativeLaunch, ctx->device) == cudaSuccess && coop &&
        cudaFuncSetAttribute(k_trif_loop, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kTrifLoopSmem) ==
            cudaSuccess &&
        cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_trif_loop, kTrifLoopThreads, kTrifLoopSmem) ==
            cudaSuccess &&
        per_sm >= 1;
    cudaGetLastError();
    return known[ctx->device] = ok;
}

struct TriFront::Impl {
    ga_ctx ctx;
    int64_t m, nnz, cap;
    const KtBatch* batch;
    int64_t ng;
    bool one_launch;                   // the loop in one cooperative launch
    DBuf<unsigned char> mem;           // everything below (as thirty allocations 35 us of host time)
    int32_t *row_of, *pcol, *oid, *orec, *sup, *f0, *f1, *efound;                            // per entry
    int32_t *deg, *upc, *H, *rd, *rh, *mark, *touched, *flip;                                // per row
    int32_t *rd1, *rd2, *rh1, *rh2, *touched1, *touched2, *flip1, *flip2, *dcur;             // (one-launch loop)
    uint8_t *h, *state;
    TriFrontState* st;
    int32_t* cntg;
    long long* pg;
    int2* seg;
    int64_t nseg;
    void* kt_scr;
    TriKt t;
    WordRanks words;
    ga_csr_s W;                        // the matrix with partitioned rows
    TriFrontArgs a;
    cudaEvent_t ready = nullptr;       // the result has been copied
    bool first = true;

    Impl(ga_ctx ctx_, ga_csr A, const KtBatch* batch_)
        : ctx(ctx_), m(A->m), nnz(A->nnz), cap(std::max<int64_t>(A->nnz, 1)), batch(batch_),
          ng(batch_ ? batch_->ngraphs : 0), one_launch(!batch_ && ctx_->device_loops && trif_loop_fits(ctx_)),
          nseg(std::max<int64_t>(cap / 8, 4096)) {
        mem = DBuf<unsigned char>(ctx, carve(nullptr));
        carve(mem.p);
        tri_kt_carve(kt_scr, m, cap, &t);
        words = WordRanks{t.bits, t.pre};
        W.m = W.n = m;
        W.nnz = nnz;
        W.rst = A->rst;
        W.col = pcol;
        W.dtype = GA_INT32;
        GA_CUDA(cudaMemsetAsync(st, 0, sizeof(TriFrontState), ctx->stream));
        if (batch) {
            GA_CUDA(cudaMemsetAsync(cntg, 0, sizeof(int32_t) * (size_t)(2 * ng), ctx->stream));
            GA_CUDA(cudaMemsetAsync(pg, 0, sizeof(long long) * (size_t)ng, ctx->stream));
        }
        a.cr = A->rst;
        a.cc = pcol;
        a.ac = A->col;
        a.row_of = row_of;
        a.crank = t.crank;
        a.rank = t.rank;
        a.ocount = t.ocount;
        a.dpos = t.dpos;
        a.oid = oid;
        a.orec = orec;
        a.sup = sup;
        a.state = state;
        a.deg = deg;
        a.upc = upc;
        a.h = h;
        a.H = H;
        a.rd = rd;
        a.rh = rh;
        a.mark = mark;
        a.touched = touched;
        a.flip = flip;
        a.f0 = f0;
        a.f1 = f1;
        a.seg = seg;
        a.efound = efound;
        a.segcap = nseg;
        a.st = st;
        a.ctr = ctx->d_counters;
        a.m = m;
        a.nnz = nnz;
        a.k = 0;
        a.gid = batch ? batch->gid : nullptr;
        a.kg = batch ? batch->kg : nullptr;
        a.nvert = batch ? batch->nvert : nullptr;
        a.done_g = batch ? batch->done_g : nullptr;
        a.iters_g = batch ? batch->iters_g : nullptr;
        a.cntg = batch ? cntg : nullptr;
        a.pg = batch ? pg : nullptr;
        a.ngraphs = ng;
        // one-launch loop: its frontiers share f0, so f1 holds segments
        a.rd1 = rd1;
        a.rd2 = rd2;
        a.rh1 = rh1;
        a.rh2 = rh2;
        a.touched1 = touched1;
        a.touched2 = touched2;
        a.flip1 = flip1;
        a.flip2 = flip2;
        a.dcur = one_launch ? dcur : nullptr;
        a.seg1 = reinterpret_cast<int2*>(f1);
        a.segcap1 = std::min<int64_t>(a.segcap, cap / 2);
        GA_CUDA(cudaEventCreateWithFlags(&ready, cudaEventDisableTiming));
    }

    // Places of the arrays from `base` on; the bytes they take.
    size_t carve(unsigned char* base) {
        size_t off = 0;
        auto take = [&](auto** p, int64_t count) {
            using E = std::remove_reference_t<decltype(**p)>;
            *p = reinterpret_cast<E*>(base + off);
            off += align256(sizeof(E) * (size_t)count);
        };
        for (int32_t** p : {&row_of, &pcol, &oid, &orec, &sup, &f0, &f1, &efound}) take(p, cap);
        for (int32_t** p : {&deg, &upc, &H, &rd, &rh, &mark, &touched, &flip}) take(p, m + 1);
        for (int32_t** p : {&rd1, &rd2, &rh1, &rh2, &touched1, &touched2, &flip1, &flip2, &dcur})
            take(p, one_launch ? m + 1 : 1);
        take(&h, m + 1);
        take(&state, cap);
        take(&st, 1);
        take(&cntg, batch ? 2 * ng : 1);
        take(&pg, batch ? ng : 1);
        take(&seg, nseg);
        kt_scr = base + off;
        return off + tri_kt_bytes(m, cap);
    }

    ~Impl() {
        if (ready) cudaEventDestroy(ready);
    }

    // The matrix as the loop stores it, its records and the counts of C_0;
    // iteration 0's supports by one listing of every triangle; the first
    // frontier.
    void begin() {
        const int grid_ent = grid_for(cap, 256, ctx->num_sms * 16);
        ga_csr_s A = W;
        A.col = const_cast<int32_t*>(a.ac);
        expand_rows(ctx, &A, row_of);
        trikt_partition(ctx, a.cr, a.ac, m, nnz, row_of, t, batch, pcol);
        k_trif_init_rows<<<grid_for(m, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(a);
        post_launch("trif_init_rows");
        if (nnz) {
            k_trif_records<<<grid_ent, 256, 0, ctx->stream>>>(a, words, t.dpos);
            post_launch("trif_records");
        }
        k_trif_init_counts<<<grid_for(std::max<int64_t>(m, ng), 256, ctx->num_sms * 2), 256, 0, ctx->stream>>>(a);
        post_launch("trif_init_counts");
        tri_kt_support(ctx, &W, sup, t, cap);
        if (nnz) {
            ProfScope ps(ctx, "trif_seed");
            k_trif_seed<<<grid_for((cap + kSeedWords - 1) / kSeedWords, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(a);
            post_launch("trif_seed");
        }
    }

    void run(int k) {
        a.k = k;
        if (first) {
            first = false;
            begin();
        } else {
            GA_REQUIRE(!batch, GA_ERR_INVALID_ARG, "a batched frontier k-truss runs one k");
            // a new k: the loop state restarts (the running work totals stay)
            ProfScope ps(ctx, "trif_seed");
            GA_CUDA(cudaMemsetAsync(st, 0, offsetof(TriFrontState, live), ctx->stream));
            if (nnz) {
                k_trif_reseed<<<grid_for((cap + kSeedWords - 1) / kSeedWords, 256, ctx->num_sms * 8), 256, 0, ctx->stream>>>(a);
                post_launch("trif_reseed");
            }
        }
        if (one_launch) {
            ProfScope ps(ctx, "ktruss_loop");
            void* args[] = {&a};
            if (cudaLaunchCooperativeKernel((const void*)k_trif_loop, dim3(ctx->num_sms), dim3(kTrifLoopThreads), args,
                                            kTrifLoopSmem, ctx->stream) == cudaSuccess) {
                post_launch("trif_loop");
                return;
            }
            // the device cannot hold the whole grid at once (part of it is set
            // aside): the captured loop serves
            cudaGetLastError();
            one_launch = false;
        }
        if (!batch) {
            k_trif_begin<<<1, 32, 0, ctx->stream>>>(a);
            post_launch("trif_begin");
        }
        // The loop's kernels read the call's parameters from a device copy and
        // have fixed grids, so the context captures the loop once per slot and
        // relaunches it on later calls.
        const int slot = batch ? kLoopSlotTriFrontBatch : kLoopSlotTriFront;
        TriFrontArgs* dargs = static_cast<TriFrontArgs*>(cached_loop_args(ctx, slot, sizeof(TriFrontArgs)));
        GA_CUDA(cudaMemcpyAsync(dargs, &a, sizeof(TriFrontArgs), cudaMemcpyHostToDevice, ctx->stream));
        const int sms = ctx->num_sms;
        const bool batched = batch != nullptr;
        ga_ctx c = ctx;
        auto body = [c, dargs, sms, batched](const LoopCtl& ctl) {
            if (batched) {
                ProfScope ps(c, "trif_mark");
                k_trif_mark<<<sms * 4, 256, 0, c->stream>>>(dargs);
                post_launch("trif_mark");
            }
            {
                ProfScope ps(c, "trif_lower");
                k_trif_lower<<<sms * kTrifLowerCtas, 128, 0, c->stream>>>(dargs);
                post_launch("trif_lower");
                k_trif_lower_seg<<<sms * kTrifLowerCtas, 128, 0, c->stream>>>(dargs);
                post_launch("trif_lower_seg");
            }
            {
                ProfScope ps(c, "trif_apply");
                k_trif_apply<<<sms * kTrifPassCtas, 256, 0, c->stream>>>(dargs);
                post_launch("trif_apply");
            }
            {
                ProfScope ps(c, "trif_flip");
                k_trif_flip<<<sms * kTrifPassCtas, 256, 0, c->stream>>>(dargs);
                post_launch("trif_flip");
            }
            ProfScope ps(c, "trif_delta");
            k_trif_delta<<<sms * 2, 256, 0, c->stream>>>(dargs, ctl);
            post_launch("trif_delta");
            if (batched) {
                k_trif_graphs<<<sms * 2, 256, 0, c->stream>>>(dargs, ctl);
                post_launch("trif_graphs");
            }
        };
        ProfScope ps(ctx, "ktruss_loop");
        run_cached_loop(ctx, slot, body, m + 1);
    }

    // Entries kept and iteration count of the last run (one wait, during
    // which the device goes on to the kept entries' places).
    int64_t result(int* iters) {
        static_assert(sizeof(TriFrontResult) <= 64, "the context's pinned words");
        GA_CUDA(cudaMemcpyAsync(ctx->h_pinned, &st->iters, sizeof(TriFrontResult), cudaMemcpyDeviceToHost,
                                ctx->stream));
        GA_CUDA(cudaEventRecord(ready, ctx->stream));
        {
            ProfScope ps(ctx, "trif_compact");
            const int64_t nw = rank_words(nnz);
            k_trif_keep<<<grid_for(nw * 32, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(a, words);
            post_launch("trif_keep");
            scan_exclusive_i32_scratch(ctx, t.pre, t.pre, nw, t.scan_scr);
        }
        GA_CUDA(cudaEventSynchronize(ready));
        TriFrontResult r;
        std::memcpy(&r, ctx->h_pinned, sizeof(r));
        GA_REQUIRE(!r.failed, GA_ERR_TIMEOUT, "k-truss: a wait inside the loop ran out");
        if (iters) *iters = r.iters;
        return (int64_t)r.ent;
    }

    // After result(): the kept entries, values one, rows in column order.
    void compact(int32_t* rst, int32_t* col, int32_t* val) {
        ProfScope ps(ctx, "trif_compact");
        k_trif_out<<<grid_for(nnz > m ? nnz : m + 1, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(a, words, col, val,
                                                                                                  rst);
        post_launch("trif_out");
    }
};

TriFront::TriFront(ga_ctx ctx, ga_csr A, const KtBatch* batch) : impl_(new Impl(ctx, A, batch)) {}

TriFront::~TriFront() { delete impl_; }

void TriFront::run(int k) { impl_->run(k); }

ga_csr TriFront::result(int* iters) {
    const int64_t kept = impl_->result(iters);
    ga_csr C = csr_alloc(impl_->ctx, impl_->m, impl_->m, kept, GA_INT32);
    try {
        impl_->compact(C->rst, C->col, static_cast<int32_t*>(C->val));
    } catch (...) {
        csr_destroy(impl_->ctx, C);
        throw;
    }
    C->unit = 1;
    C->sym = 1;
    return C;
}

}  // namespace ga
