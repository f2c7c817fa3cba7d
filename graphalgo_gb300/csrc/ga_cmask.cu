// Complemented-mask SpGEMM C<!M> = A*B (new pattern, sorted columns) and the
// "naive" masked product built on it (full product, then a mask gather).
//
// Two passes over the same per-row machinery, as the reference does
// (matrix_la.h:800-891): a symbolic pass counts each row's output columns,
// a prefix sum gives the row starts, a numeric pass fills columns and values.
// One CTA per row (grid-stride). A row whose product count P_i is at most
// kHashMax uses a shared-memory hash of its product columns; the surviving
// keys (not in M's row) are sorted with a block bitonic sort. Longer rows are
// processed in column windows of kWin columns with a dense shared-memory
// accumulator and bitmap, which yields sorted output directly.
//
// Products with at most kNarrowCols columns (the frontier of a batched search:
// one column per source) take the narrow path below instead where it pays
// (narrow_pays).
#include "ga_device.cuh"

namespace ga {

constexpr int kCmThreads = 256;
constexpr int kCmWarps = kCmThreads / 32;
constexpr int kHashMax = 2048;          // products handled by the hash path
constexpr int kHashBitsMax = 12;        // 4096-entry table
constexpr int kWin = 4096;              // columns per dense window

template <typename T>
struct CmArgs {
    const int32_t* ar; const int32_t* ac; const T* av;
    const int32_t* br; const int32_t* bc; const T* bv;
    const int32_t* mr; const int32_t* mc;  // mr == nullptr: no mask
    int64_t m;
    const int64_t* flops;  // P_i per row
    int32_t* cnt;          // symbolic output
    const int32_t* cr;     // numeric: row starts
    int32_t* cc; T* cv;    // numeric outputs
};

__global__ void k_cm_flops(const int32_t* __restrict__ ar, const int32_t* __restrict__ ac,
                           const int32_t* __restrict__ br, int64_t m, int64_t* __restrict__ flops) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < m; i += warps) {
        long long f = 0;
        for (int32_t t = ar[i] + lane; t < ar[i + 1]; t += 32) {
            int32_t k = ac[t];
            f += br[k + 1] - br[k];
        }
        f = warp_sum<long long>(f);
        if (lane == 0) flops[i] = f;
    }
}

__device__ __forceinline__ bool in_mask(const int32_t* mc, int32_t mb, int32_t me, int32_t c) {
    int n = me - mb;
    int p = lower_bound_i32(mc + mb, n, c);
    return p < n && mc[mb + p] == c;
}

// Visit every product (col, a*b) of row i whose column lies in [lo, hi],
// flattened over the lanes of each warp; warps take groups of 32 A entries.
template <bool CLIP, typename T, typename Fn>
__device__ __forceinline__ void foreach_product(const CmArgs<T>& p, int64_t i, int32_t lo, int32_t hi, int* s_incl,
                                                int* s_off, T* s_a, Fn fn) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int32_t ab = p.ar[i], ae = p.ar[i + 1];
    for (int32_t g = ab + wid * 32; g < ae; g += kCmWarps * 32) {
        int32_t t = g + lane;
        int len = 0;
        int32_t bs = 0;
        T a = (T)0;
        if (t < ae) {
            int32_t k = p.ac[t];
            a = p.av[t];
            bs = p.br[k];
            int32_t be = p.br[k + 1];
            if (CLIP) {
                int n = be - bs;
                int l = lower_bound_i32(p.bc + bs, n, lo);
                int h = upper_bound_i32(p.bc + bs, n, hi);
                be = bs + h;
                bs = bs + l;
            }
            len = be - bs;
        }
        int incl = warp_incl_scan(len);
        int total = __shfl_sync(0xffffffffu, incl, 31);
        s_incl[lane] = incl;
        s_off[lane] = bs - (incl - len);
        s_a[lane] = a;
        __syncwarp();
        int q = 0;
        for (int x = lane; x < total; x += 32) {
            while (s_incl[q] <= x) ++q;
            int32_t j = x + s_off[q];
            fn(__ldg(p.bc + j), s_a[q], j);
        }
        __syncwarp();
    }
}

// Block-wide exclusive scan of one int per thread.
__device__ __forceinline__ int block_scan_int(int v, int* warp_tot, int* total) {
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    int x = warp_incl_scan(v);
    if (lane == 31) warp_tot[wid] = x;
    __syncthreads();
    if (wid == 0) {
        int w = lane < kCmWarps ? warp_tot[lane] : 0;
        int y = warp_incl_scan(w);
        if (lane < kCmWarps) warp_tot[lane] = y - w;
        if (lane == kCmWarps - 1) *total = y;
    }
    __syncthreads();
    int r = x - v + warp_tot[wid];
    __syncthreads();
    return r;
}

template <typename T>
struct CmSmem {
    static constexpr size_t hash_bytes = (size_t)(1 << kHashBitsMax) * (sizeof(int32_t) + sizeof(T)) +
                                         (size_t)(1 << kHashBitsMax) * (sizeof(int32_t) + sizeof(T));
    static constexpr size_t win_bytes = (size_t)kWin * sizeof(T) + (size_t)(kWin / 32) * sizeof(uint32_t);
    static constexpr size_t scratch = (size_t)kCmWarps * 32 * (2 * sizeof(int) + sizeof(T));
    static constexpr size_t total = (hash_bytes > win_bytes ? hash_bytes : win_bytes) + scratch;
};

template <bool NUMERIC, typename T>
__global__ void __launch_bounds__(kCmThreads) k_cmask(CmArgs<T> p) {
    extern __shared__ __align__(16) unsigned char smem[];
    using SM = CmSmem<T>;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned char* scr = smem + (SM::total - SM::scratch);
    int* s_incl = reinterpret_cast<int*>(scr) + wid * 32;
    int* s_off = reinterpret_cast<int*>(scr) + kCmWarps * 32 + wid * 32;
    T* s_a = reinterpret_cast<T*>(scr + (size_t)kCmWarps * 32 * 2 * sizeof(int)) + wid * 32;
    __shared__ int s_wt[32];
    __shared__ int s_total;
    __shared__ int32_t s_lo, s_hi;
    (void)lane;

    for (int64_t i = blockIdx.x; i < p.m; i += gridDim.x) {
        const int64_t P = p.flops[i];
        const int32_t mb = p.mr ? p.mr[i] : 0, me = p.mr ? p.mr[i + 1] : 0;
        if (P == 0) {
            if (!NUMERIC && threadIdx.x == 0) p.cnt[i] = 0;
            continue;
        }
        if (P <= kHashMax) {
            // ---------------------------------------------------- hash path
            int bits = 6;
            while ((1 << bits) < 2 * P) ++bits;
            const int TBL = 1 << bits;
            const uint32_t mask = TBL - 1;
            int32_t* keys = reinterpret_cast<int32_t*>(smem);
            T* vals = reinterpret_cast<T*>(smem + (size_t)(1 << kHashBitsMax) * sizeof(int32_t));
            int32_t* sk = reinterpret_cast<int32_t*>(smem + (size_t)(1 << kHashBitsMax) * (sizeof(int32_t) + sizeof(T)));
            T* sv = reinterpret_cast<T*>(reinterpret_cast<unsigned char*>(sk) + (size_t)(1 << kHashBitsMax) * sizeof(int32_t));
            for (int t = threadIdx.x; t < TBL; t += blockDim.x) {
                keys[t] = kEmpty;
                if (NUMERIC) vals[t] = (T)0;
            }
            __syncthreads();
            foreach_product<false, T>(p, i, 0, 0, s_incl, s_off, s_a, [&](int32_t c, T a, int32_t j) {
                uint32_t h = hash_col(c) >> (32 - bits);
                while (true) {
                    int32_t prev = atomicCAS(&keys[h], kEmpty, c);
                    if (prev == kEmpty || prev == c) {
                        if (NUMERIC) atomicAdd(&vals[h], a * __ldg(p.bv + j));
                        break;
                    }
                    h = (h + 1) & mask;
                }
            });
            __syncthreads();
            // survivors: present and not in the mask row; TBL <= 4096 so each
            // of the 256 threads owns at most 16 consecutive entries
            const int per = (TBL + kCmThreads - 1) / kCmThreads;
            const int t0 = threadIdx.x * per;
            int mine = 0;
            for (int u = 0; u < per; ++u) {
                int t = t0 + u;
                if (t < TBL && keys[t] != kEmpty && !in_mask(p.mc, mb, me, keys[t])) ++mine;
            }
            int pos = block_scan_int(mine, s_wt, &s_total);
            const int count = s_total;
            if (!NUMERIC) {
                if (threadIdx.x == 0) p.cnt[i] = count;
                __syncthreads();
                continue;
            }
            for (int u = 0; u < per; ++u) {
                int t = t0 + u;
                if (t < TBL && keys[t] != kEmpty && !in_mask(p.mc, mb, me, keys[t])) {
                    sk[pos] = keys[t];
                    sv[pos] = vals[t];
                    ++pos;
                }
            }
            int p2 = 1;
            while (p2 < count) p2 <<= 1;
            __syncthreads();
            for (int t = count + threadIdx.x; t < p2; t += blockDim.x) sk[t] = INT32_MAX;
            __syncthreads();
            for (int k = 2; k <= p2; k <<= 1) {
                for (int j = k >> 1; j > 0; j >>= 1) {
                    for (int t = threadIdx.x; t < p2; t += blockDim.x) {
                        int x = t ^ j;
                        if (x > t) {
                            bool up = (t & k) == 0;
                            int32_t a = sk[t], b = sk[x];
                            if ((a > b) == up) {
                                sk[t] = b; sk[x] = a;
                                T va = sv[t]; sv[t] = sv[x]; sv[x] = va;
                            }
                        }
                    }
                    __syncthreads();
                }
            }
            const int32_t o = p.cr[i];
            for (int t = threadIdx.x; t < count; t += blockDim.x) {
                p.cc[o + t] = sk[t];
                p.cv[o + t] = sv[t];
            }
            __syncthreads();
        } else {
            // ------------------------------------------- windowed dense path
            T* acc = reinterpret_cast<T*>(smem);
            uint32_t* bits = reinterpret_cast<uint32_t*>(smem + (size_t)kWin * sizeof(T));
            // column range of the products
            if (threadIdx.x == 0) { s_lo = INT32_MAX; s_hi = -1; }
            __syncthreads();
            {
                int32_t lo = INT32_MAX, hi = -1;
                for (int32_t t = p.ar[i] + threadIdx.x; t < p.ar[i + 1]; t += blockDim.x) {
                    int32_t k = p.ac[t];
                    int32_t b = p.br[k], e = p.br[k + 1];
                    if (e > b) {
                        lo = min(lo, p.bc[b]);
                        hi = max(hi, p.bc[e - 1]);
                    }
                }
                atomicMin(&s_lo, lo);
                atomicMax(&s_hi, hi);
            }
            __syncthreads();
            const int32_t lo_all = s_lo, hi_all = s_hi;
            int running = 0;
            for (int64_t w0 = lo_all; w0 <= hi_all; w0 += kWin) {
                const int32_t wlo = (int32_t)w0;
                const int32_t whi = (int32_t)((w0 + kWin - 1) < (int64_t)hi_all ? (w0 + kWin - 1) : (int64_t)hi_all);
                for (int t = threadIdx.x; t < kWin / 32; t += blockDim.x) bits[t] = 0u;
                if (NUMERIC)
                    for (int t = threadIdx.x; t < kWin; t += blockDim.x) acc[t] = (T)0;
                __syncthreads();
                foreach_product<true, T>(p, i, wlo, whi, s_incl, s_off, s_a, [&](int32_t c, T a, int32_t j) {
                    int d = c - wlo;
                    atomicOr(&bits[d >> 5], 1u << (d & 31));
                    if (NUMERIC) atomicAdd(&acc[d], a * __ldg(p.bv + j));
                });
                __syncthreads();
                // drop the mask row's columns inside the window
                if (p.mr) {
                    int n = me - mb;
                    int s = lower_bound_i32(p.mc + mb, n, wlo);
                    for (int q = s + threadIdx.x; q < n; q += blockDim.x) {
                        int32_t c = p.mc[mb + q];
                        if (c > whi) break;
                        int d = c - wlo;
                        atomicAnd(&bits[d >> 5], ~(1u << (d & 31)));
                    }
                }
                __syncthreads();
                // kWin/32 = 128 words over 256 threads: one word per thread
                uint32_t word = threadIdx.x < kWin / 32 ? bits[threadIdx.x] : 0u;
                int pos = block_scan_int(__popc(word), s_wt, &s_total);
                const int wcount = s_total;
                if (NUMERIC) {
                    const int32_t o = p.cr[i] + running + pos;
                    int r = 0;
                    while (word) {
                        int b = __ffs(word) - 1;
                        word &= word - 1;
                        int d = threadIdx.x * 32 + b;
                        p.cc[o + r] = wlo + d;
                        p.cv[o + r] = acc[d];
                        ++r;
                    }
                }
                running += wcount;
                __syncthreads();
            }
            if (!NUMERIC && threadIdx.x == 0) p.cnt[i] = running;
            __syncthreads();
        }
    }
}

// ------------------------------------------------------------- narrow path
// B with at most kNarrowCols columns, handled in blocks of 64: a row's pattern
// inside a block is one 64-bit word. The symbolic pass ORs the words of the B
// rows an A row selects (8 bytes per A entry, no product is visited) and drops
// the mask row's; the numeric pass gives every lane two columns of the block,
// transposes the words of 32 B rows across the warp, and each lane walks the
// rows that hold its columns, their values placed by popcounts. The sums stay
// in registers: no hash table, no sort, no atomics.
//
// What bounds it: the chain of gathers per 32 A entries (column, word, B row
// start, values) from the L2, and in FP64 the adder (2 lanes per clock and SM
// whether one lane of the warp is active or 32), which is why the lanes walk
// their own lists: visiting the B rows one by one with a lane per column left
// 3 of 32 lanes active and took 1,520 us for the level below. A row with more
// than kNarrowHeavy entries is cut into pieces of kNarrowPiece that separate
// CTAs sum (with 512-thread CTAs and pieces of 2,048 the numeric pass took 171
// us: the rows of a CTA wait for its longest); the last piece to finish adds
// the pieces in order.
//
// One breadth-first level of 64 sources on R-MAT 16 (complemented product,
// 1.9M A entries, 2.1e5 frontier entries, 30 % of the pairs masked): 157 us
// (words 12, symbolic 37, numeric 108); the per-row hash path below takes
// 4,350 us. The line at kNarrowCols, the largest batch of sources: frontier
// density 0.002 / 0.05 / 0.3 on the same graph, whole call, this path against
// the hash and window path: 64 columns 163 / 232 / 453 against 1,400 / 4,860 /
// 9,074 us; 256 columns 297 / 592 / 1,505 against 2,397 / 8,072 / 17,819 us;
// 1,024 columns 874 / 2,045 / 5,681 against 4,707 / 15,473 / 54,951 us.
constexpr int kNarrowCols = 1024;
constexpr int kNarrowThreads = 512;      // symbolic pass
constexpr int kNarrowWarps = kNarrowThreads / 32;
constexpr int kNarrowSumThreads = 128;   // numeric pass: small CTAs, a long row holds up few others
constexpr int kNarrowSumWarps = kNarrowSumThreads / 32;
constexpr int kNarrowHeavy = 256;
constexpr int kNarrowPiece = 512;

struct NarrowTask {
    int32_t row, piece;   // kNarrowPiece entries of the row
    int32_t first, count; // the row's pieces: places first .. first + count - 1 of the partial sums
};

struct NarrowArgs {
    const unsigned long long* bbits;  // [block][row of B]: columns of the block
    const int32_t* bpos;              // [block][row of B]: position of the first of them
    unsigned long long* pat;          // [block][row of A]: columns of the result
    int64_t bm;                       // rows of B
    int blocks;
    NarrowTask* tasks;
    int32_t* ntask;
    int32_t* done;                    // per place: pieces finished (at the row's first place)
    void* part;                       // partial sums, 64 per place and block
};

// Words of a matrix's rows, one warp per row.
__global__ void k_row_bits(const int32_t* __restrict__ rst, const int32_t* __restrict__ col, int64_t m, int blocks,
                           unsigned long long* __restrict__ bits, int32_t* __restrict__ pos) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < m; i += warps) {
        const int32_t e = rst[i + 1];
        int32_t b = rst[i];
        for (int x = 0; x < blocks; ++x) {
            uint32_t lo = 0, hi = 0;
            int32_t q = b;
            bool more = true;
            while (more) {  // warp-uniform
                const int32_t c = q + lane < e ? col[q + lane] - x * 64 : 64;
                if (c < 32) lo |= 1u << c;
                else if (c < 64) hi |= 1u << (c - 32);
                const int in = __popc(__ballot_sync(0xffffffffu, c < 64));
                q += in;
                more = in == 32;
            }
            lo = __reduce_or_sync(0xffffffffu, lo);
            hi = __reduce_or_sync(0xffffffffu, hi);
            if (lane == 0) {
                bits[(int64_t)x * m + i] = ((unsigned long long)hi << 32) | lo;
                pos[(int64_t)x * m + i] = b;
            }
            b = q;
        }
    }
}

// Row of warp `wid` in CTA b: warp w's rows are the w-th run of gridDim.x
// rows, shifted, so that neither neighbouring rows nor rows a power of two
// apart (both are where an R-MAT graph has its hubs) share a CTA.
__device__ __forceinline__ int64_t narrow_row(int wid) {
    return (int64_t)wid * gridDim.x + (blockIdx.x + 1571u * (unsigned)wid) % gridDim.x;
}

// OR over the warp of a 64-bit word.
__device__ __forceinline__ unsigned long long warp_or64(unsigned long long w) {
    const uint32_t lo = __reduce_or_sync(0xffffffffu, (uint32_t)w);
    const uint32_t hi = __reduce_or_sync(0xffffffffu, (uint32_t)(w >> 32));
    return ((unsigned long long)hi << 32) | lo;
}

// Result pattern and count of every row; the pieces of long rows.
__global__ void __launch_bounds__(kNarrowThreads) k_narrow_symbolic(NarrowArgs a, const int32_t* __restrict__ ar,
                                                                    const int32_t* __restrict__ ac,
                                                                    const int32_t* __restrict__ mr,
                                                                    const int32_t* __restrict__ mc, int64_t m,
                                                                    int32_t* __restrict__ cnt) {
    __shared__ unsigned long long s_or[kNarrowWarps][kNarrowCols / 64];
    __shared__ int2 s_row[kNarrowWarps];
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    const int64_t i = narrow_row(wid);
    const int32_t ab = i < m ? ar[i] : 0, ae = i < m ? ar[i + 1] : 0;
    const bool heavy = ae - ab > kNarrowHeavy;
    if (lane < kNarrowCols / 64) s_or[wid][lane] = 0ull;
    if (lane == 0) s_row[wid] = make_int2(ab, ae);
    __syncthreads();
    // long rows: all warps, one row after the other
    for (int h = 0; h < kNarrowWarps; ++h) {
        const int32_t hb = s_row[h].x, he = s_row[h].y;
        if (he - hb <= kNarrowHeavy) continue;
        for (int x = 0; x < a.blocks; ++x) {
            const unsigned long long* bb = a.bbits + (int64_t)x * a.bm;
            unsigned long long w = 0;
#pragma unroll 4
            for (int32_t t = hb + (int32_t)threadIdx.x; t < he; t += kNarrowThreads) w |= __ldg(bb + __ldg(ac + t));
            w = warp_or64(w);
            if (lane == 0 && w) atomicOr(&s_or[h][x], w);
        }
    }
    __syncthreads();
    if (i >= m) return;
    int32_t mq = mr ? mr[i] : 0;
    const int32_t me = mr ? mr[i + 1] : 0;
    int n = 0;
    for (int x = 0; x < a.blocks; ++x) {
        const unsigned long long* bb = a.bbits + (int64_t)x * a.bm;
        unsigned long long w = 0, mw = 0;
        if (heavy) {
            w = s_or[wid][x];
        } else {
#pragma unroll 4
            for (int32_t t = ab + lane; t < ae; t += 32) w |= __ldg(bb + __ldg(ac + t));
            w = warp_or64(w);
        }
        bool more = mq < me;
        while (more) {  // warp-uniform: the mask row's columns in this block
            const int32_t c = mq + lane < me ? mc[mq + lane] - x * 64 : 64;
            if (c < 64) mw |= 1ull << c;
            const int in = __popc(__ballot_sync(0xffffffffu, c < 64));
            mq += in;
            more = in == 32;
        }
        w &= ~warp_or64(mw);
        if (lane == 0) a.pat[(int64_t)x * m + i] = w;
        n += __popcll(w);
    }
    if (lane != 0) return;
    cnt[i] = n;
    if (heavy && n) {
        const int pieces = (ae - ab + kNarrowPiece - 1) / kNarrowPiece;
        const int first = atomicAdd(a.ntask, pieces);
        a.done[first] = 0;
        for (int c = 0; c < pieces; ++c) a.tasks[first + c] = NarrowTask{(int32_t)i, c, first, pieces};
    }
}

// Sums of the lane's two columns of block x (lane, lane + 32) over the A
// entries [t0, t1), groups of 32 at stride `step`. s_at / s_lo / s_hi / s_a:
// 32 entries each in shared memory for the warp.
template <typename T>
__device__ __forceinline__ void narrow_sums(const CmArgs<T>& p, const NarrowArgs& a, int x, int32_t t0, int32_t t1,
                                            int32_t step, unsigned long long pw, int32_t* s_at, uint32_t* s_lo,
                                            uint32_t* s_hi, T* s_a, T& acc0, T& acc1) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    const unsigned long long* bb = a.bbits + (int64_t)x * a.bm;
    for (int32_t g = t0; g < t1; g += step) {
        const int32_t t = g + lane;
        unsigned long long w = 0;
        int32_t k = 0;
        if (t < t1) {
            k = __ldg(p.ac + t);
            w = __ldg(bb + k);
        }
        const bool hit = (w & pw) != 0ull;
        if (__ballot_sync(FULL, hit) == 0u) continue;
        __syncwarp();  // the last group's lists are read
        T av = (T)1;
        if (hit) {
            s_at[lane] = __ldg(a.bpos + (int64_t)x * a.bm + k);
            s_a[lane] = av = p.av[t];
        }
        // a group of ones (an unweighted graph) needs no products
        const bool ones = __all_sync(FULL, av == (T)1);
        s_lo[lane] = (uint32_t)w;
        s_hi[lane] = (uint32_t)(w >> 32);
        __syncwarp();
        // bit j: B row j of the group holds column `lane`; bit 32 + j: column lane + 32
        const uint32_t m0 = warp_transpose_bits((uint32_t)(w & pw));
        const uint32_t m1 = warp_transpose_bits((uint32_t)((w & pw) >> 32));
        unsigned long long mine = ((unsigned long long)m1 << 32) | m0;
        while (mine) {
            T v[4], f[4];
            bool on[4], high[4];
#pragma unroll
            for (int h = 0; h < 4; ++h) {
                on[h] = mine != 0ull;
                high[h] = false;
                if (on[h]) {
                    const int j = __ffsll((long long)mine) - 1;
                    mine &= mine - 1;
                    high[h] = j >= 32;
                    const int r = j & 31;
                    const int off = high[h] ? __popc(s_lo[r]) + __popc(s_hi[r] & lt) : __popc(s_lo[r] & lt);
                    v[h] = __ldg(p.bv + s_at[r] + off);
                    f[h] = s_a[r];
                }
            }
#pragma unroll
            for (int h = 0; h < 4; ++h)
                if (on[h]) {
                    const T c = high[h] ? acc1 : acc0;
                    const T s = ones ? c + v[h] : mul_add_separate<T>(c, f[h], v[h]);
                    if (high[h]) acc1 = s;
                    else acc0 = s;
                }
        }
    }
}

// Row i's entries of block x, whose first result entry is at o.
template <typename T>
__device__ __forceinline__ void narrow_store(const CmArgs<T>& p, int x, int32_t o, unsigned long long pw, T acc0,
                                             T acc1) {
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u, lo = (uint32_t)pw, hi = (uint32_t)(pw >> 32);
    if (lo >> lane & 1u) {
        const int32_t q = o + __popc(lo & lt);
        p.cc[q] = x * 64 + lane;
        p.cv[q] = acc0;
    }
    if (hi >> lane & 1u) {
        const int32_t q = o + __popc(lo) + __popc(hi & lt);
        p.cc[q] = x * 64 + 32 + lane;
        p.cv[q] = acc1;
    }
}

template <typename T>
__global__ void __launch_bounds__(kNarrowSumThreads) k_narrow_numeric(CmArgs<T> p, NarrowArgs a) {
    __shared__ T s_acc[kNarrowSumWarps][64];
    __shared__ int32_t s_at[kNarrowSumWarps][32];
    __shared__ uint32_t s_lo[kNarrowSumWarps][32], s_hi[kNarrowSumWarps][32];
    __shared__ T s_a[kNarrowSumWarps][32];
    __shared__ bool s_last;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    T* part = static_cast<T*>(a.part);
    const int ntask = *a.ntask;
    for (int it = blockIdx.x; it < ntask; it += gridDim.x) {
        const NarrowTask task = a.tasks[it];
        const int32_t ab = p.ar[task.row] + task.piece * kNarrowPiece;
        const int32_t ae = min(p.ar[task.row + 1], ab + kNarrowPiece);
        for (int x = 0; x < a.blocks; ++x) {
            const unsigned long long pw = a.pat[(int64_t)x * p.m + task.row];
            T acc0 = (T)0, acc1 = (T)0;
            if (pw)
                narrow_sums<T>(p, a, x, ab + wid * 32, ae, kNarrowSumThreads, pw, s_at[wid], s_lo[wid], s_hi[wid],
                               s_a[wid], acc0, acc1);
            s_acc[wid][lane] = acc0;
            s_acc[wid][32 + lane] = acc1;
            __syncthreads();
            if (threadIdx.x < 64) {
                T sum = (T)0;
                for (int w = 0; w < kNarrowSumWarps; ++w) sum += s_acc[w][threadIdx.x];
                part[((int64_t)it * a.blocks + x) * 64 + threadIdx.x] = sum;
            }
            __syncthreads();
        }
        // the row's last piece to finish adds them all, in order
        if (threadIdx.x < 64) __threadfence();
        __syncthreads();
        if (threadIdx.x == 0) s_last = atomicAdd(a.done + task.first, 1) == task.count - 1;
        __syncthreads();
        if (s_last && wid == 0) {
            __threadfence();
            int32_t o = p.cr[task.row];
            for (int x = 0; x < a.blocks; ++x) {
                const unsigned long long pw = a.pat[(int64_t)x * p.m + task.row];
                T acc0 = (T)0, acc1 = (T)0;
                for (int c = 0; c < task.count; ++c) {
                    const T* q = part + ((int64_t)(task.first + c) * a.blocks + x) * 64;
                    acc0 += __ldcg(q + lane);
                    acc1 += __ldcg(q + 32 + lane);
                }
                narrow_store<T>(p, x, o, pw, acc0, acc1);
                o += __popcll(pw);
            }
        }
        __syncthreads();
    }
    const int64_t i = narrow_row(wid);
    if (i >= p.m) return;
    const int32_t ab = p.ar[i], ae = p.ar[i + 1];
    int32_t o = p.cr[i];
    if (ae - ab > kNarrowHeavy || o == p.cr[i + 1]) return;
    for (int x = 0; x < a.blocks; ++x) {
        const unsigned long long pw = a.pat[(int64_t)x * p.m + i];
        if (pw == 0ull) continue;
        T acc0 = (T)0, acc1 = (T)0;
        narrow_sums<T>(p, a, x, ab, ae, 32, pw, s_at[wid], s_lo[wid], s_hi[wid], s_a[wid], acc0, acc1);
        narrow_store<T>(p, x, o, pw, acc0, acc1);
        o += __popcll(pw);
    }
}

// Whether the narrow path is the faster one, in nanoseconds of either beyond
// what both need. The words are made for every row of B and of A whether an
// entry of A meets it or not, so few rows of A against a tall B are the general
// path's, which takes a CTA per row of A that has entries. B of 10^6 x 64 / 10^6
// x 1,024 with two entries per row, A of 256 rows of 64 entries: 130 / 984 us by
// words, 60 / 61 by rows; of 2,048: 136 / 1,006 and 133 / 160; 16,384: 182 /
// 1,269 and 728 / 883; B of 20,000 x 64 / 1,024: 75 / 146 and 62 / 61, 76 / 144
// and 139 / 159, 123 / 369 and 728 / 883. Rows in pieces are summed twice: 2,048
// rows of 1,024 entries, B of 20,000 x 1,024, 1,109 and 747. Nearly empty
// matrices of 2 x 10^6 rows, 0.05 entries each, 64 / 256 / 1,024 columns: 1,180 /
// 1,781 / 3,973 and 3,600.
static bool narrow_pays(const ga_csr_s& A, const ga_csr_s& B) {
    const double rows = (double)std::min(A.m, A.nnz), nnz = (double)A.nnz, tall = (double)B.m;
    const double by_rows = 22.0 * rows + 0.11 * nnz * (1.0 + (double)B.nnz / std::max(tall, 1.0));
    const double per_entry = A.nnz > A.m * kNarrowHeavy ? 0.04 : 0.02;
    const double by_words = 1e4 + (double)((B.n + 63) / 64) * (0.08 * tall + 0.02 * (double)A.m + per_entry * nnz);
    return by_words < by_rows;
}

template <typename T>
static ga_csr cmask_narrow(ga_ctx ctx, ga_csr A, ga_csr B, CmArgs<T> p) {
    const int64_t m = A->m;
    const int blocks = (int)((B->n + 63) / 64);
    const size_t places = (size_t)(A->nnz / kNarrowPiece + A->nnz / kNarrowHeavy + 1);
    DBuf<unsigned long long> bbits(ctx, (size_t)B->m * blocks), pat(ctx, (size_t)m * blocks);
    DBuf<int32_t> bpos(ctx, (size_t)B->m * blocks), cnt(ctx, (size_t)m + 1), rst(ctx, (size_t)m + 2);
    DBuf<NarrowTask> tasks(ctx, places);
    DBuf<int32_t> done(ctx, places);
    int32_t* ntask = rst.p + m + 1;  // behind the entries' number: one copy reads both
    NarrowArgs a{bbits.p, bpos.p, pat.p, B->m, blocks, tasks.p, ntask, done.p, nullptr};
    const unsigned grid = (unsigned)((m + kNarrowWarps - 1) / kNarrowWarps);
    {
        ProfScope ps(ctx, "cmask_symbolic");
        GA_CUDA(cudaMemsetAsync(ntask, 0, sizeof(int32_t), ctx->stream));
        k_row_bits<<<grid_for(B->m * 32, 256, ctx->num_sms * 64), 256, 0, ctx->stream>>>(B->rst, B->col, B->m, blocks,
                                                                                         bbits.p, bpos.p);
        post_launch("cmask_row_bits");
        k_narrow_symbolic<<<grid, kNarrowThreads, 0, ctx->stream>>>(a, A->rst, A->col, p.mr, p.mc, m, cnt.p);
        post_launch("cmask_narrow_symbolic");
    }
    scan_exclusive_i32(ctx, cnt.p, rst.p, m);
    int32_t* h = reinterpret_cast<int32_t*>(ctx->h_pinned);
    GA_CUDA(cudaMemcpyAsync(h, rst.p + m, 2 * sizeof(int32_t), cudaMemcpyDeviceToHost, ctx->stream));
    GA_CUDA(cudaStreamSynchronize(ctx->stream));
    const int64_t nnz = h[0];
    DBuf<T> part(ctx, (size_t)h[1] * blocks * 64);  // partial sums of the pieces that there are
    a.part = part.p;
    ga_csr C = csr_alloc(ctx, m, B->n, nnz, A->dtype);
    try {
        GA_CUDA(cudaMemcpyAsync(C->rst, rst.p, sizeof(int32_t) * (m + 1), cudaMemcpyDeviceToDevice, ctx->stream));
        if (nnz) {
            p.cr = C->rst; p.cc = C->col; p.cv = static_cast<T*>(C->val);
            ProfScope ps(ctx, "cmask_numeric");
            k_narrow_numeric<T><<<(unsigned)((m + kNarrowSumWarps - 1) / kNarrowSumWarps), kNarrowSumThreads, 0,
                                  ctx->stream>>>(p, a);
            post_launch("cmask_narrow_numeric");
        }
    } catch (...) {
        csr_destroy(ctx, C);
        throw;
    }
    return C;
}

template <typename T>
static ga_csr cmask_typed(ga_ctx ctx, ga_csr A, ga_csr B, const int32_t* mr, const int32_t* mc) {
    CmArgs<T> p;
    p.ar = A->rst; p.ac = A->col; p.av = static_cast<const T*>(A->val);
    p.br = B->rst; p.bc = B->col; p.bv = static_cast<const T*>(B->val);
    p.mr = mr; p.mc = mc; p.m = A->m;
    p.flops = nullptr; p.cnt = nullptr; p.cr = nullptr; p.cc = nullptr; p.cv = nullptr;
    if (A->m > 0 && B->n >= 1 && B->n <= kNarrowCols && narrow_pays(*A, *B)) {
        // Where its words (per 64 columns 12 bytes a row of B and 8 a row of A,
        // empty rows too) or its partial sums do not fit in memory, the path
        // below serves: it needs 16 bytes a row of A.
        try {
            return cmask_narrow<T>(ctx, A, B, p);
        } catch (const Error& e) {
            if (e.code != GA_ERR_OOM) throw;
        }
    }
    DBuf<int64_t> flops(ctx, (size_t)A->m + 1);
    DBuf<int32_t> cnt(ctx, (size_t)A->m + 1);
    p.flops = flops.p; p.cnt = cnt.p;
    {
        ProfScope ps(ctx, "cmask_flops");
        k_cm_flops<<<grid_for(A->m * 32, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(A->rst, A->col, B->rst, A->m,
                                                                                        flops.p);
        post_launch("cmask_flops");
    }
    const size_t smem = CmSmem<T>::total;
    GA_CUDA(cudaFuncSetAttribute(k_cmask<false, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    GA_CUDA(cudaFuncSetAttribute(k_cmask<true, T>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 1;
    GA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k_cmask<true, T>, kCmThreads, smem));
    if (per_sm < 1) per_sm = 1;
    const int grid = (int)std::min<int64_t>(A->m > 0 ? A->m : 1, (int64_t)ctx->num_sms * per_sm);
    if (A->m > 0) {
        ProfScope ps(ctx, "cmask_symbolic");
        k_cmask<false, T><<<grid, kCmThreads, smem, ctx->stream>>>(p);
        post_launch("cmask_symbolic");
    }
    DBuf<int32_t> rst(ctx, (size_t)A->m + 1);
    if (A->m > 0) scan_exclusive_i32(ctx, cnt.p, rst.p, A->m);
    else GA_CUDA(cudaMemsetAsync(rst.p, 0, sizeof(int32_t), ctx->stream));
    int64_t nnz = read_i32(ctx, rst.p + A->m);
    ga_csr C = csr_alloc(ctx, A->m, B->n, nnz, A->dtype);
    try {
        GA_CUDA(cudaMemcpyAsync(C->rst, rst.p, sizeof(int32_t) * (A->m + 1), cudaMemcpyDeviceToDevice, ctx->stream));
        if (nnz) {
            p.cr = C->rst; p.cc = C->col; p.cv = static_cast<T*>(C->val);
            ProfScope ps(ctx, "cmask_numeric");
            k_cmask<true, T><<<grid, kCmThreads, smem, ctx->stream>>>(p);
            post_launch("cmask_numeric");
        }
    } catch (...) {
        csr_destroy(ctx, C);
        throw;
    }
    return C;
}

ga_csr mxm_cmask(ga_ctx ctx, ga_csr A, ga_csr B, ga_csr M) {
    GA_REQUIRE(A->n == B->m, GA_ERR_SHAPE, "cmask: A.n != B.m");
    GA_REQUIRE(!M || (M->m == A->m && M->n == B->n), GA_ERR_SHAPE, "cmask: mask shape differs from A*B");
    GA_REQUIRE(A->dtype == B->dtype, GA_ERR_DTYPE, "cmask: A and B dtypes differ");
    const int32_t* mr = M ? M->rst : nullptr;
    const int32_t* mc = M ? M->col : nullptr;
    ga_csr C = nullptr;
    switch (A->dtype) {
    case GA_INT32: C = cmask_typed<int32_t>(ctx, A, B, mr, mc); break;
    case GA_INT64: C = cmask_typed<unsigned long long>(ctx, A, B, mr, mc); break;
    case GA_FP32: C = cmask_typed<float>(ctx, A, B, mr, mc); break;
    case GA_FP64: C = cmask_typed<double>(ctx, A, B, mr, mc); break;
    case GA_UINT8: fail(GA_ERR_DTYPE, "cmask: uint8 values are not supported");
    }
    C->dtype = A->dtype;
    return C;
}

// ----------------------------------------------------------- naive variant
// C<M> = A*B by the full product followed by a gather of the mask entries
// (mxmm_naive, include/matrix_la.h:1139-1277): each mask entry binary-searches
// its column in the product row; absent entries are 0.
template <typename T>
__global__ void k_mask_gather(const int32_t* __restrict__ pr, const int32_t* __restrict__ pc,
                              const T* __restrict__ pv, const int32_t* __restrict__ mr,
                              const int32_t* __restrict__ mc, int64_t m, T* __restrict__ cv) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < m; i += warps) {
        int32_t b = pr[i], n = pr[i + 1] - b;
        for (int32_t q = mr[i] + lane; q < mr[i + 1]; q += 32) {
            int32_t c = mc[q];
            int p = lower_bound_i32(pc + b, n, c);
            cv[q] = (p < n && pc[b + p] == c) ? pv[b + p] : (T)0;
        }
    }
}

void naive_masked_into(ga_ctx ctx, ga_csr A, ga_csr B, ga_csr M, void* d_cvals) {
    GA_REQUIRE(A->dtype != GA_UINT8, GA_ERR_DTYPE, "naive: uint8 values are not supported");
    ProfScope ps(ctx, "mxm_naive");
    ga_csr P = mxm_cmask(ctx, A, B, nullptr);
    try {
        GA_DISPATCH_DTYPE(A->dtype, T, {
            k_mask_gather<T><<<grid_for(M->m * 32, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(
                P->rst, P->col, static_cast<const T*>(P->val), M->rst, M->col, M->m, static_cast<T*>(d_cvals));
        });
        post_launch("mask_gather");
    } catch (...) {
        csr_destroy(ctx, P);
        throw;
    }
    csr_destroy(ctx, P);
}

}  // namespace ga

using namespace ga;

extern "C" int ga_mxm_cmask(ga_ctx ctx, ga_csr A, ga_csr B, ga_csr M, ga_csr* C) {
    if (!ctx || !A || !B || !M || !C) return GA_ERR_INVALID_ARG;
    *C = nullptr;
    GA_API_BODY(ctx, *C = mxm_cmask(ctx, A, B, M));
}
