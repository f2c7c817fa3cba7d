// Masked SpGEMM C<M> = A*B (structural mask, C has M's pattern).
//
// Design (one pass, no symbolic phase: the output pattern is M's):
//  1. k_row_bin computes each output row's mask length m_i and Gustavson
//     product count P_i = sum_{k in A_i} nnz(B_k). Rows with an
//     empty mask are skipped, rows without products get explicit zeros, short
//     light rows (m_i <= warp_slots, P_i <= warp_max_flops or a limit of the
//     product's own) go to a warp queue, all others to a CTA queue as windows
//     of at most kCtaSlots mask slots spanning fewer than kWinCols columns
//     (heavy rows first, the heaviest in more windows).
//  2. k_mxm_masked: a persistent kernel (one wave of CTAs sized by occupancy)
//     drains the CTA queue, then every warp drains the warp queue. The
//     accumulator is indexed by mask slot and lives in shared memory.
//     Column -> slot lookup per variant:
//       GA_MSA, : a dense bitmap of the window's mask columns in shared memory
//       GA_MCA    (the reference MSA keeps a dense state array over the
//                 columns, matrix_la.h:681-749); a set bit is resolved to its
//                 slot as the word's first slot plus a popcount (the
//                 slot base is kept per 32-column word). Warp rows use a
//                 4096-bit hashed filter and a 512-entry hash table. The
//                 accumulator is the mask row's entries, which is MCA's too:
//                 the reference MCA finds the entry by walking the mask row
//                 (matrix_la.h:625-632), here the rank of the set bit is it.
//                 A binary search of the mask row behind the same filters
//                 was slower at every size tried: a 50,021 x 40,009 product of
//                 1e8 products under 24-entry mask rows 914 us against 631 in
//                 FP64 and 721 against 417 in int32, 1,000 x 1,000 with 10
//                 entries per row 141 against 128, R-MAT 16 support 2,764
//                 against 1,162, 32-entry rows under 2-entry masks 1,947
//                 against 945;
//       GA_HEAP : sorted merge of each B row against the mask row
//                 (replaces the priority-queue merge,
//                 matrix_la.h:1030-1084): lanes take 32 A entries; a B row
//                 with few entries inside the window is merged by its lane,
//                 a longer one is cut into 32 slices merged by one lane
//                 each (the mask side gallops), and a B row far longer
//                 than the mask row is merged by the whole warp, 32
//                 columns against 32, galloping over the B runs that
//                 cannot meet the mask.
//     Work distribution inside a CTA item: warps take the row's A entries 32
//     at a time; B rows of up to kLongSeg entries (32 when the A row is too
//     short to occupy every warp) are flattened over the
//     warp's lanes (warp scan of the lengths, lanes walk the flattened index);
//     longer B rows (hubs) go to a shared list and are cut into kChunk-entry
//     pieces that all warps of the CTA stream coalesced.
// Integer results are exact and equal across variants; floating-point sums
// are accumulated with shared-memory atomics (order not fixed).
#include "ga_device.cuh"

#include <algorithm>
#include <type_traits>

namespace ga {

constexpr int kMxmThreads = 512;
constexpr int kMxmWarps = kMxmThreads / 32;
// Mask slots per CTA work item. Half as many of 8 bytes: the
// third CTA fits on an SM then (75 KB each instead of 90), FP64 products of
// 200,000 x 200,000 under 8-entry mask rows 1,695 -> 1,484 us, 50,021 x
// 40,009 under 32-entry rows 2,195 -> 2,104.
template <typename A> constexpr int kCtaSlots = sizeof(A) == 8 ? 2048 : 4096;
// Mask slots per warp row, and those up to which a warp's table holds columns:
// with accumulators of 8 bytes three CTAs' tables of 256 do not fit on an SM, and
// longer rows take one of slots (MD_SLOTS), in a kernel of its own for masks of
// more than kSlotsMean entries per row on average. As CTA items, which take 22
// ns however few products a row has, such rows were ten times slower: FP64
// products of 200,000 rows under 129 / 180 / 256 mask entries, 100 products per
// row 4,440 / 4,560 / 4,710 us, so 323 / 400 / 516; 4,800 per row 11,480 / 11,570
// / 11,680 and 2,140 / 2,540 / 3,430. That kernel is 3 to 6 % slower where all
// rows are shorter (60 / 120 entries, 900 products per row 456 / 553 us, so 478 /
// 579), and up to 20 % where few rows are longer and these have many products
// (50,021 x 40,009 under power-law rows of 24 entries on average 509 and 624;
// of 67: 224 and 188). Merging has no table: all its rows up to 256 are a warp's,
// unless there are so few that CTAs take them side by side (1,000 rows of 900
// products 41 us by CTAs, 50 by warps; 30,000 rows 354 and 206).
constexpr int kWarpSlots = 256;
template <typename A> constexpr int kColumnSlots = sizeof(A) == 8 ? 128 : 256;
constexpr int kSlotsMean = 64;
constexpr int kFewRows = 12;   // rows per SM
constexpr int kNoSlot = 255;
constexpr int kLeastCtaSlots = 2048;
constexpr int kWinCols = 1 << 17;          // column span of a CTA work item
constexpr int kWinWords = kWinCols / 32;   // dense bitmap words
constexpr int kWarpTblBits = 9;            // warp-row hash table: 512 entries
constexpr int kFilterBits = 12;            // warp-row filter: 4096 bits
constexpr int kDotTask = 8;                // hybrid form: mask entries per inner-product task
// Bin thresholds (rows above warp_max_flops products go to a CTA; CTA items
// of rows with at least heavy_flops products are scheduled first) and the
// persistent grid size are runtime parameters (ga_ctx tune, set by options
// or the autotuner).
constexpr int kLongSeg = 256;              // B rows longer than this are shared by the CTA
constexpr int kShortARow = kMxmThreads;    // A rows with fewer entries leave warps idle in phase A:
constexpr int kLongSegShort = 32;          // their B rows longer than this are shared instead
constexpr int kLongCap = 1024;             // long B rows listed per item
constexpr int kChunk = 1024;               // entries per long-row piece

struct MxmQueue {
    int32_t warp_count;
    int32_t heavy_count;   // CTA items at the front of the item array
    int32_t normal_count;  // CTA items at the back
    int32_t warp_next;
    int32_t cta_next;
    int32_t dot_count;     // hybrid form: inner-product tasks listed
    int32_t split_count;   // windows that heavy rows were split into
};

// Shares of the whole that a row is split into, and the products it has at least.
struct BinSplit {
    float shares;
    long long least;
};

template <typename T, typename A>
struct MxmArgs {
    const int32_t* ar; const int32_t* ac; const T* av;
    const int32_t* br; const int32_t* bc; const T* bv;
    const int32_t* mr; const int32_t* mc;
    // row ends: row i of A is [ar[i], are[i]), and so on
    const int32_t* are; const int32_t* bre; const int32_t* mre;
    // the mask rows that the work counters count (the whole mask where only
    // part of it is evaluated)
    const int32_t* cmr; const int32_t* cme;
    bool clip;  // B rows are cut to the mask row's span (part of the mask: worth two searches per B row)
    T* cv;
    int64_t m;
    MxmQueue* q;
    int32_t* warp_rows;
    int4* cta_items;          // (row, first slot, end slot, unused)
    int32_t cta_cap;
    unsigned long long* ctr;  // context work counters (GA_CTR_*)
    int64_t warp_max_flops, heavy_flops;
    int32_t warp_slots;       // mask entries that a warp row has at most
    bool small;               // warp_max_flops is only a bound, and heavy rows are split
    BinSplit split;
    // hybrid form: rows whose inner-product work (sum over mask entries of
    // min(|A_i|, |B^T_j|)) times hybrid_ratio is below their Gustavson work
    // are listed in dot_tasks (row, first mask entry; count in the queue),
    // kDotTask mask entries per task, for the inner-product kernel
    const int32_t* btr;  // B^T row starts (nullptr: no hybrid)
    int2* dot_tasks;
    int64_t hybrid_ratio;
};

__global__ void k_reset_queue(MxmQueue* q) {
    if (threadIdx.x == 0) {
        q->warp_count = 0; q->heavy_count = 0; q->normal_count = 0;
        q->warp_next = 0; q->cta_next = 0; q->dot_count = 0; q->split_count = 0;
    }
}

// ------------------------------------------------------------------ binning
constexpr int kBinThreads = 256;

// Products of A entries [t0, t1) at stride `step`, this thread's share.
template <typename T, typename A>
__device__ __forceinline__ long long bin_products(const MxmArgs<T, A>& p, int32_t t0, int32_t t1, int32_t step) {
    long long f = 0;
#pragma unroll 4
    for (int32_t t = t0; t < t1; t += step) {
        const int32_t k = __ldg(p.ac + t);
        f += __ldg(p.bre + k) - __ldg(p.br + k);
    }
    return f;
}

// Products up to which a short row is a warp's, in a product that is small for
// the device. A warp takes about 1.6 ns per product; a CTA 0.1 ns, but 5 us per
// row, and rows wait when there are more of them than CTAs. With the rows of f
// products or more sent to CTAs, at most total / f of them, the slowest on
// either side is fastest near f = kWarpShare * sqrt(total). Every CTA estimates
// the total from the same kSamples of A's entries, while it reads its first rows
// (where all rows are alike, it is 0.5 to 2 us lost; with four times as many
// samples 2 to 5). With 32,768 at every size, and so: supports of R-MAT 9, 10, 12, 13 (0.27M to 19M
// products) 64 / 168 / 273 / 398 and 34 / 49 / 109 / 114 us, of 1,000 vertices
// with 180 neighbours 314 and 123, MSA k-truss of R-MAT 11 960 and 402. With
// kWarpShare 2.6 and 4.0 R-MAT 13 takes 136 and 197, with 1.1 5,000 vertices
// with 80 neighbours take 219 instead of 171.
constexpr int kSamples = kBinThreads;
constexpr float kWarpShare = 1.6f;
constexpr long long kWarpLeast = 1024;

// This thread's sample: the loads are under way while the first rows are read.
struct BinSample {
    int32_t b = 0, e = 0;
    int64_t nnz, count;
};
template <typename T, typename A>
__device__ __forceinline__ BinSample bin_sample(const MxmArgs<T, A>& p) {
    BinSample s;
    const int64_t first = p.ar[0];
    s.nnz = (int64_t)p.ar[p.m] - first;
    s.count = s.nnz < kSamples ? s.nnz : kSamples;
    if (threadIdx.x < s.count) {
        const int32_t k = __ldg(p.ac + first + threadIdx.x * s.nnz / s.count);
        s.b = __ldg(p.br + k);
        s.e = __ldg(p.bre + k);
    }
    return s;
}

// Products of the whole, estimated. All threads of the CTA.
__device__ __forceinline__ float bin_total(const BinSample& s) {
    __shared__ long long part[kBinThreads / 32];
    long long f = warp_sum<long long>(s.e - s.b);
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = f;
    __syncthreads();
    f = 0;
    for (int w = 0; w < kBinThreads / 32; ++w) f += part[w];
    return s.count ? (float)f * ((float)s.nnz / (float)s.count) : 0.0f;
}

// A row of more products than its share of the whole is cut into as many
// windows as it holds shares, each of them an item that meets only the part of
// the B rows inside it: as one item, the heaviest row of R-MAT 16 (1.4M
// products) keeps a CTA busy for nearly as long as the rest takes the whole
// device. Items of half a share and more start first. Support of R-MAT 14, 15,
// 17 by MSA 353 / 584 / 1,012 and 331 / 559 / 938 us, of R-MAT 12, 14, 16 (4 per
// vertex) by merging 322 / 1,143 / 1,014 and 224 / 742 / 545; MSA k-truss of
// R-MAT 16 6.5 and 5.7 ms. MSA rows of fewer than 131,072 products are not
// worth another look at A's row (R-MAT 12 from 32,768 on: 98 and 111 us). Of
// 608, 912, 1,216 and 1,824 shares MSA is best with 912 (R-MAT 14: 314, 331,
// 332, 355; R-MAT 16: 993, 988, 955, 965), merging, which takes three times as
// long per product, with 1,824 (R-MAT 15: 1,459, 1,472, 1,397, 1,257).
constexpr BinSplit kSplit = {912.0f, 131072}, kSplitMerge = {1824.0f, 32768};
constexpr int kSplitSlots = 32;             // mask slots that a window has at least
constexpr int kSplitItems = 4096;           // windows of all split rows together

// The bins of `take` rows per warp at a time (up to 32; fewer when the matrix
// has not that many rows for every resident warp). Queue places are reserved
// for the rows together: with one atomic per row, a union of a million short rows
// took 700 us, nearly all of it on the counter (512 30-NN graphs' triangle
// counts; now 180 us). A warp's rows lie far apart and at no power of two
// (a power-law graph's hubs sit together or a power of two apart), and rows
// of more than kBinLong entries are summed by the whole CTA (R-MAT 18
// support: 236 -> 69 us).
constexpr int kBinLong = 1024;

template <typename T, typename A>
__global__ void __launch_bounds__(kBinThreads) k_row_bin(MxmArgs<T, A> p, int take) {
    __shared__ int32_t s_long[kBinThreads];           // the CTA's long rows: thread that holds each
    __shared__ long long s_sum[kBinThreads];          // products of the row held by each thread
    __shared__ int2 s_range[kBinThreads];
    __shared__ int s_nlong, s_at;
    __shared__ int s_short[kBinThreads / 32];
    __shared__ unsigned long long s_work[3];
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    if (threadIdx.x < 3) s_work[threadIdx.x] = 0;
    long long warp_max = p.small ? -1 : p.warp_max_flops, split = INT64_MAX, heavy_min = p.heavy_flops;
    BinSample sample;
    if (p.small) sample = bin_sample(p);
    unsigned long long my_flops = 0, my_mask = 0, my_entries = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&p.ctr[GA_CTR_LAUNCHES], 1ull);
        atomicAdd(&p.ctr[GA_CTR_ROWS], (unsigned long long)p.m);
    }
    const int64_t groups = (p.m + take - 1) / take;  // lane l's rows: the l-th run of `groups` rows, shifted
    const int64_t step = (int64_t)gridDim.x * (kBinThreads / 32);
    for (int64_t g0 = (int64_t)blockIdx.x * (kBinThreads / 32); g0 < groups; g0 += step) {
        const int64_t g = g0 + wid;
        int64_t i = p.m;
        if (g < groups && lane < take) i = take == 1 ? g : (g + 1571ll * lane) % groups + (int64_t)lane * groups;
        int32_t mb = 0, me = 0, ab = 0, ae = 0, count = 0;
        if (i < p.m) {
            mb = p.mr[i];
            me = p.mre[i];
            ab = p.ar[i];
            ae = p.are[i];
            count = p.cme[i] - p.cmr[i];
        }
        const bool live = me > mb, counted = count > 0;
        if (counted) my_mask += (unsigned long long)count;
        my_entries += (unsigned long long)(ae - ab);
        if (threadIdx.x == 0) s_nlong = 0;
        __syncthreads();
        const bool is_long = counted && ae - ab > kBinLong;
        if (is_long) {
            s_long[atomicAdd(&s_nlong, 1)] = threadIdx.x;
            s_range[threadIdx.x] = make_int2(ab, ae);
            s_sum[threadIdx.x] = 0;
        }
        __syncthreads();
        for (int x = 0; x < s_nlong; ++x) {
            const int th = s_long[x];
            long long f = bin_products(p, s_range[th].x + (int32_t)threadIdx.x, s_range[th].y, kBinThreads);
            f = warp_sum<long long>(f);
            if (lane == 0 && f) atomicAdd(reinterpret_cast<unsigned long long*>(&s_sum[th]), (unsigned long long)f);
        }
        __syncthreads();
        long long f = is_long ? s_sum[threadIdx.x] : 0;
        for (unsigned rows = __ballot_sync(FULL, counted && !is_long); rows; rows &= rows - 1) {
            const int r = __ffs(rows) - 1;
            const int32_t b = __shfl_sync(FULL, ab, r), e = __shfl_sync(FULL, ae, r);
            const long long fr = warp_sum<long long>(bin_products(p, b + lane, e, 32));
            if (lane == r) f = fr;
        }
        if (warp_max < 0) {
            const float total = bin_total(sample);
            warp_max = min((long long)p.warp_max_flops, max(kWarpLeast, (long long)(kWarpShare * sqrtf(total))));
            split = max(p.split.least, (long long)(total / p.split.shares));
            heavy_min = min(heavy_min, split / 2);
        }
        // rows without products: explicit zeros
        for (unsigned rows = __ballot_sync(FULL, live && f == 0); rows; rows &= rows - 1) {
            const int r = __ffs(rows) - 1;
            const int32_t b = __shfl_sync(FULL, mb, r), e = __shfl_sync(FULL, me, r);
            for (int32_t q = b + lane; q < e; q += 32) p.cv[q] = (T)0;
        }
        const int32_t mi = me - mb;
        bool todo = live && f != 0;
        my_flops += (unsigned long long)f;
        if (p.btr) {
            // inner-product work of each row; the cheaper form takes it
            for (unsigned rows = __ballot_sync(FULL, todo); rows; rows &= rows - 1) {
                const int r = __ffs(rows) - 1;
                const int32_t b = __shfl_sync(FULL, mb, r), e = __shfl_sync(FULL, me, r);
                const int32_t an = __shfl_sync(FULL, ae - ab, r);
                const long long fr = __shfl_sync(FULL, f, r);
                long long dsum = 0;
                for (int32_t q = b + lane; q < e; q += 32) {
                    const int32_t j = p.mc[q];
                    const int32_t bn = p.btr[j + 1] - p.btr[j];
                    dsum += an < bn ? an : bn;
                }
                dsum = warp_sum<long long>(dsum);
                if (dsum * p.hybrid_ratio < fr) {
                    const int ntask = (e - b + kDotTask - 1) / kDotTask;
                    int first = 0;
                    if (lane == 0) first = atomicAdd(&p.q->dot_count, ntask);
                    first = __shfl_sync(FULL, first, 0);
                    const int row = __shfl_sync(FULL, (int)i, r);
                    for (int t = lane; t < ntask; t += 32) p.dot_tasks[first + t] = make_int2(row, b + t * kDotTask);
                    if (lane == r) todo = false;
                }
            }
        }
        // warp rows
        const bool short_row = todo && mi <= p.warp_slots && f <= warp_max;
        unsigned set = __ballot_sync(FULL, short_row);
        if (lane == 0) s_short[wid] = __popc(set);
        __syncthreads();
        if (wid == 0) {
            const int mine = lane < kBinThreads / 32 ? s_short[lane] : 0, incl = warp_incl_scan(mine);
            if (lane < kBinThreads / 32) s_short[lane] = incl - mine;
            if (lane == 31 && incl) s_at = atomicAdd(&p.q->warp_count, incl);
        }
        __syncthreads();
        if (short_row) p.warp_rows[s_at + s_short[wid] + __popc(set & ((1u << lane) - 1u))] = (int32_t)i;
        // CTA items: rows of one window together, the others window by window
        const bool cta_row = todo && !short_row;
        const int32_t* mcol = p.mc + mb;
        const bool heavy = f >= heavy_min;
        const bool one = cta_row && mi <= kCtaSlots<A> && f <= split && mcol[mi - 1] - mcol[0] < kWinCols;
        for (int h = 0; h < 2; ++h) {
            const bool in = one && heavy == (h == 0);
            set = __ballot_sync(FULL, in);
            if (!set) continue;
            int pos = 0;
            if (lane == 0) pos = atomicAdd(h == 0 ? &p.q->heavy_count : &p.q->normal_count, __popc(set));
            pos = __shfl_sync(FULL, pos, 0) + __popc(set & ((1u << lane) - 1u));
            if (in) p.cta_items[h == 0 ? pos : p.cta_cap - 1 - pos] = make_int4((int)i, 0, mi, 0);
        }
        if (cta_row && !one) {
            int s0 = 0, slots = kCtaSlots<A>;
            if (f > split) {
                const int windows = (int)min(f / split + 1, (long long)(mi + kSplitSlots - 1) / kSplitSlots);
                const int each = (mi + windows - 1) / windows;
                if (each < slots && atomicAdd(&p.q->split_count, windows) + windows <= kSplitItems) slots = each;
            }
            while (s0 < mi) {
                int s1 = min(mi, s0 + slots);
                const int32_t c0 = mcol[s0];
                if (mcol[s1 - 1] - c0 >= kWinCols) {
                    const int64_t lim = (int64_t)c0 + (kWinCols - 1);
                    s1 = s0 + upper_bound_i32(mcol + s0, s1 - s0, (int32_t)(lim < INT32_MAX ? lim : INT32_MAX));
                }
                int pos;
                if (heavy) pos = atomicAdd(&p.q->heavy_count, 1);
                else pos = p.cta_cap - 1 - atomicAdd(&p.q->normal_count, 1);
                p.cta_items[pos] = make_int4((int)i, s0, s1, 0);
                s0 = s1;
            }
        }
    }
    // one addition per CTA and counter, as for the warp rows' places: with the
    // warps' own, 4,786 rows took 14 us instead of 7.4
    my_flops = warp_sum<unsigned long long>(my_flops);
    my_mask = warp_sum<unsigned long long>(my_mask);
    my_entries = warp_sum<unsigned long long>(my_entries);
    if (lane == 0) {
        if (my_flops) atomicAdd(&s_work[0], my_flops);
        if (my_mask) atomicAdd(&s_work[1], my_mask);
        if (my_entries) atomicAdd(&s_work[2], my_entries);
    }
    __syncthreads();
    if (threadIdx.x < 3 && s_work[threadIdx.x])
        atomicAdd(&p.ctr[threadIdx.x == 0 ? GA_CTR_PRODUCTS : threadIdx.x == 1 ? GA_CTR_MASK_ENTRIES : GA_CTR_A_ENTRIES],
                  s_work[threadIdx.x]);
}

// ------------------------------------------------------------------ lookups
// How a product's column finds its mask slot: MD_DENSE in CTA items, MD_HASHED
// or MD_SLOTS in warp rows; MD_MERGE merges whole B rows instead.
enum { MD_DENSE = 0, MD_HASHED = 1, MD_MERGE = 2, MD_SLOTS = 3 };

// The mask columns of one work item, staged in shared memory.
struct SlotView {
    const int32_t* mcol;    // MD_MERGE, MD_SLOTS: sorted mask columns
    const uint32_t* bits;   // MD_DENSE: bitmap over [lo, lo + kWinCols)
    const uint16_t* wbase;  // MD_DENSE: slot of the first mask column of each bitmap word
    const uint32_t* filt;   // MD_HASHED, MD_SLOTS: 4096-bit filter of hashed columns
    const int32_t* hkeys;   // MD_HASHED: open-addressing table (2^kWarpTblBits)
    const uint8_t* hslot;   // MD_HASHED: their slots; MD_SLOTS: the table itself (kNoSlot: none)
    int ns;
    int32_t lo, hi;
};

// Word of the window's bitmap that column c lies in, and that word moved up so
// that c's bit is the highest: its sign is the test, and what is below it the
// rank. Columns outside the window's span read the guard word behind the
// bitmap; inside it only mask columns have their bit set. (A range check, a
// shift and a mask for each: R-MAT 18 support by halves 6,450 us, so 5,640;
// R-MAT 16 1,160 and 1,000. Testing a lane's eight columns before any hit, or
// looping over its hits, is slower at 1,062 to 1,230.)
__device__ __forceinline__ uint32_t dense_word(const SlotView& v, int32_t c, uint32_t* d) {
    *d = min((uint32_t)(c - v.lo), (uint32_t)kWinCols);
    return __funnelshift_l(0u, v.bits[*d >> 5], ~*d);
}

template <int MD>
__device__ __forceinline__ int slot_of(const SlotView& v, int32_t c) {
    if (MD == MD_DENSE) {
        // dense state over the window: a set bit is a mask column, and its
        // slot is the word's first slot plus the set bits below it
        uint32_t d;
        const uint32_t w = dense_word(v, c, &d);
        return (int32_t)w < 0 ? (int)v.wbase[d >> 5] + __popc(w) - 1 : -1;
    } else {
        const uint32_t h = hash_col(c);
        const uint32_t f = h >> (32 - kFilterBits);
        if (!((v.filt[f >> 5] >> (f & 31)) & 1u)) return -1;
        const uint32_t mask = (1u << kWarpTblBits) - 1u;
        uint32_t pos = h >> (32 - kWarpTblBits);
        if (MD == MD_SLOTS) {
            if (c == v.hi) return v.ns - 1;  // slot 255 would be kNoSlot: the last column is not in the table
            int slot = v.hslot[pos];
            while (slot != kNoSlot && v.mcol[slot] != c) {
                pos = (pos + 1) & mask;
                slot = v.hslot[pos];
            }
            return slot == kNoSlot ? -1 : slot;
        }
        // One way out of the loop. With a return for the hit and one for the
        // empty place inside it, the code that nvcc 13.0 makes left lanes that
        // hit at their first place out of later rounds of the row while others
        // probed on (8 of 36,000 rows under 200 to 256 mask entries came out
        // wrong, always the same; barriers around the loop did not help).
        int32_t key = v.hkeys[pos];
        while (key != c && key != kEmpty) {
            pos = (pos + 1) & mask;
            key = v.hkeys[pos];
        }
        return key == c ? (int)v.hslot[pos] : -1;
    }
}

// Enters the slot of column c into a table of slots (used: a bit per place, as
// bytes cannot be claimed by themselves).
__device__ __forceinline__ void slot_insert(uint32_t* used, uint8_t* hslot, int32_t c, int slot) {
    uint32_t pos = hash_col(c) >> (32 - kWarpTblBits);
    while (true) {
        const uint32_t bit = 1u << (pos & 31);
        if (!(atomicOr(&used[pos >> 5], bit) & bit)) break;
        pos = (pos + 1) & ((1u << kWarpTblBits) - 1u);
    }
    hslot[pos] = (uint8_t)slot;
}

// Value modes: VM 0 general, 1 B's values are all ones (no B value loads),
// 2 A's and B's values are all ones (every product is 1: no value loads or
// multiplies at all; int32 only).
// B value of entry j in the accumulator type.
template <int VM, typename T, typename A>
__device__ __forceinline__ A bval(const MxmArgs<T, A>& p, int32_t j) {
    return VM >= 1 ? (A)1 : to_acc<T, A>(__ldg(p.bv + j));
}

// Adds a product to the slot of column c, if the mask has one.
template <int MD, typename A>
__device__ __forceinline__ void add_product(const SlotView& v, A* acc, int32_t c, A prod) {
    const int slot = slot_of<MD>(v, c);
    if (slot >= 0) atomic_add_acc<A>(&acc[slot], prod);
}
// The same with the product of a and b. In FP64 it is formed for the lanes of
// a hit only: a multiplication costs the SM 16 cycles, however many lanes
// need it, and most products miss the mask (1e8 products under 24-entry mask
// rows 685 -> 664 us, under 32-entry rows 2,315 -> 2,165). In the other types
// it is formed beforehand, which is 1 to 3 % faster.
template <int MD, typename A>
__device__ __forceinline__ void add_product(const SlotView& v, A* acc, int32_t c, A a, A b) {
    if (!std::is_same<A, double>::value) return add_product<MD, A>(v, acc, c, a * b);
    const int slot = slot_of<MD>(v, c);
    if (slot >= 0) atomic_add_acc<A>(&acc[slot], a * b);
}
// The same for a B value b of segment q, whose A value is staged in s_a.
template <int MD, int VM, typename A>
__device__ __forceinline__ void add_segment_product(const SlotView& v, A* acc, int32_t c, const A* s_a, int q, A b) {
    if (VM >= 1) add_product<MD, A>(v, acc, c, VM == 2 ? (A)1 : s_a[q]);
    else if (!std::is_same<A, double>::value) add_product<MD, A>(v, acc, c, s_a[q] * b);
    else {
        const int slot = slot_of<MD>(v, c);
        if (slot >= 0) atomic_add_acc<A>(&acc[slot], s_a[q] * b);
    }
}

// Four consecutive values starting at a 16-byte aligned index.
template <typename T> struct Vec4 { T x, y, z, w; };
template <typename T>
__device__ __forceinline__ Vec4<T> load4(const T* ptr) {
    Vec4<T> r;
    if (sizeof(T) == 4) {
        const int4 t = __ldg(reinterpret_cast<const int4*>(ptr));
        memcpy(&r, &t, 16);
    } else if (sizeof(T) == 8) {
        const int4 a = __ldg(reinterpret_cast<const int4*>(ptr));
        const int4 b = __ldg(reinterpret_cast<const int4*>(ptr) + 1);
        memcpy(&r, &a, 16);
        memcpy(reinterpret_cast<char*>(&r) + 16, &b, 16);
    } else {
        r.x = __ldg(ptr); r.y = __ldg(ptr + 1); r.z = __ldg(ptr + 2); r.w = __ldg(ptr + 3);
    }
    return r;
}

// B-row range of A entry t, optionally clipped to the item's column window.
template <typename T, typename A>
__device__ __forceinline__ void b_range(const MxmArgs<T, A>& p, int32_t t, bool clip, int32_t lo, int32_t hi,
                                        int32_t& bs, int32_t& be) {
    const int32_t k = __ldg(p.ac + t);
    bs = __ldg(p.br + k);
    be = __ldg(p.bre + k);
    if (clip) {
        const int n = be - bs;
        const int l = lower_bound_i32(p.bc + bs, n, lo);
        const int h = upper_bound_i32(p.bc + bs, n, hi);
        be = bs + h;
        bs = bs + l;
    }
}

// Flattened products of the 32 A entries starting at t_first (one per lane).
// Non-empty B rows are compacted; for each window of 32 consecutive product
// indices the segment ends falling inside it form one 32-bit mask (a warp OR
// reduction), so every lane finds its B row with a popcount - no per-lane
// search loop. Lanes whose B row is long may hand it to the CTA's long list.
// Returns the number of products it processed (warp-uniform).
template <int MD, int VM, typename T, typename A, bool PUSH>
__device__ __forceinline__ int group_products(const MxmArgs<T, A>& p, int32_t t_first, int32_t t_end, bool clip,
                                              const SlotView& v, A* acc, int* s_incl, int* s_off, A* s_a,
                                              int* s_nlong, int32_t* s_lbs, int32_t* s_lend, A* s_la,
                                              int long_seg = kLongSeg) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int32_t t = t_first + lane;
    int len = 0;
    int32_t bs = 0;
    A av = (A)0;
    if (t < t_end) {
        int32_t be;
        b_range(p, t, clip, v.lo, v.hi, bs, be);
        av = VM == 2 ? (A)1 : to_acc<T, A>(__ldg(p.av + t));
        len = be - bs;
        if (PUSH && len > long_seg) {
            const int slot = atomicAdd(s_nlong, 1);
            if (slot < kLongCap) {
                s_lbs[slot] = bs;
                s_lend[slot] = be;
                s_la[slot] = av;
                len = 0;
            }
        }
    }
    const unsigned nz = __ballot_sync(FULL, len > 0);
    if (nz == 0) return 0;
    const int nseg = __popc(nz);
    const int incl = warp_incl_scan(len);
    const int total = __shfl_sync(FULL, incl, 31);
    if (len > 0) {
        const int rank = __popc(nz & ((1u << lane) - 1u));
        s_incl[rank] = incl;
        s_off[rank] = bs - (incl - len);
        if (VM != 2) s_a[rank] = av;
    }
    __syncwarp();
    const int my_end = lane < nseg ? s_incl[lane] - 1 : INT32_MAX;  // last product of segment `lane`
    const unsigned lt = (1u << lane) - 1u;
    int q_base = 0;
    int base = 0;
    for (; base + 32 < total; base += 64) {
        const int e0 = my_end - base, e1 = my_end - base - 32;
        const unsigned bm0 = __reduce_or_sync(FULL, (e0 >= 0 && e0 < 32) ? (1u << e0) : 0u);
        const unsigned bm1 = __reduce_or_sync(FULL, (e1 >= 0 && e1 < 32) ? (1u << e1) : 0u);
        const int q0 = q_base + __popc(bm0 & lt);
        const int q1 = q_base + __popc(bm0) + __popc(bm1 & lt);
        const int x1 = base + 32 + lane;
        const int32_t j0 = base + lane + s_off[q0];
        const int32_t c0 = __ldg(p.bc + j0);
        const A b0 = bval<VM, T, A>(p, j0);
        int32_t c1 = 0;
        A b1 = (A)0;
        if (x1 < total) {
            const int32_t j1 = x1 + s_off[q1];
            c1 = __ldg(p.bc + j1);
            b1 = bval<VM, T, A>(p, j1);
        }
        add_segment_product<MD, VM, A>(v, acc, c0, s_a, q0, b0);
        if (x1 < total) add_segment_product<MD, VM, A>(v, acc, c1, s_a, q1, b1);
        q_base += __popc(bm0) + __popc(bm1);
    }
    if (base < total) {
        const int e0 = my_end - base;
        const unsigned bm0 = __reduce_or_sync(FULL, (e0 >= 0 && e0 < 32) ? (1u << e0) : 0u);
        const int x = base + lane;
        if (x < total) {
            const int q = q_base + __popc(bm0 & lt);
            const int32_t j = x + s_off[q];
            add_segment_product<MD, VM, A>(v, acc, __ldg(p.bc + j), s_a, q, bval<VM, T, A>(p, j));
        }
    }
    __syncwarp();
    return total;
}

// Stream B entries [j0, j1) of one row with scalar head/tail and a
// 16-byte vector body (columns, and values unless they are all ones).
template <int MD, int VM, typename T, typename A>
__device__ __forceinline__ void stream_row(const MxmArgs<T, A>& p, const SlotView& v, A* acc, int32_t j0,
                                           int32_t j1, A a) {
    const int lane = threadIdx.x & 31;
    int32_t ja = (j0 + 3) & ~3;
    if (ja > j1) ja = j1;
    if (j0 + lane < ja) add_product<MD, A>(v, acc, __ldg(p.bc + j0 + lane), a, bval<VM, T, A>(p, j0 + lane));
    const int32_t groups = (j1 - ja) >> 2;
    int32_t g = lane;
    for (; g + 32 < groups; g += 64) {
        const int32_t j = ja + 4 * g, jy = j + 128;
        const Vec4<int32_t> x = load4<int32_t>(p.bc + j);
        const Vec4<int32_t> y = load4<int32_t>(p.bc + jy);
        if (VM >= 1) {
            add_product<MD, A>(v, acc, x.x, a); add_product<MD, A>(v, acc, x.y, a);
            add_product<MD, A>(v, acc, x.z, a); add_product<MD, A>(v, acc, x.w, a);
            add_product<MD, A>(v, acc, y.x, a); add_product<MD, A>(v, acc, y.y, a);
            add_product<MD, A>(v, acc, y.z, a); add_product<MD, A>(v, acc, y.w, a);
        } else {
            const Vec4<T> bx = load4<T>(p.bv + j);
            const Vec4<T> by = load4<T>(p.bv + jy);
            add_product<MD, A>(v, acc, x.x, a, to_acc<T, A>(bx.x));
            add_product<MD, A>(v, acc, x.y, a, to_acc<T, A>(bx.y));
            add_product<MD, A>(v, acc, x.z, a, to_acc<T, A>(bx.z));
            add_product<MD, A>(v, acc, x.w, a, to_acc<T, A>(bx.w));
            add_product<MD, A>(v, acc, y.x, a, to_acc<T, A>(by.x));
            add_product<MD, A>(v, acc, y.y, a, to_acc<T, A>(by.y));
            add_product<MD, A>(v, acc, y.z, a, to_acc<T, A>(by.z));
            add_product<MD, A>(v, acc, y.w, a, to_acc<T, A>(by.w));
        }
    }
    if (g < groups) {
        const int32_t j = ja + 4 * g;
        const Vec4<int32_t> x = load4<int32_t>(p.bc + j);
        if (VM >= 1) {
            add_product<MD, A>(v, acc, x.x, a); add_product<MD, A>(v, acc, x.y, a);
            add_product<MD, A>(v, acc, x.z, a); add_product<MD, A>(v, acc, x.w, a);
        } else {
            const Vec4<T> bx = load4<T>(p.bv + j);
            add_product<MD, A>(v, acc, x.x, a, to_acc<T, A>(bx.x));
            add_product<MD, A>(v, acc, x.y, a, to_acc<T, A>(bx.y));
            add_product<MD, A>(v, acc, x.z, a, to_acc<T, A>(bx.z));
            add_product<MD, A>(v, acc, x.w, a, to_acc<T, A>(bx.w));
        }
    }
    const int32_t jt = ja + 4 * groups;
    if (jt + lane < j1) add_product<MD, A>(v, acc, __ldg(p.bc + jt + lane), a, bval<VM, T, A>(p, jt + lane));
}

// First index in [lo, hi) of a sorted array whose value is >= key (hi if
// none), found by the whole warp with 32 probes per step: the first step
// probes the ends of the next 32 runs of 32 entries (a short skip costs two
// steps), later steps split what is left 32 ways. GLOBAL: the array is in
// global memory (read-only path), else in shared memory. Warp-uniform
// arguments and result.
template <bool GLOBAL>
__device__ __forceinline__ int32_t warp_lower_bound(const int32_t* a, int32_t lo, int32_t hi, int32_t key) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    int64_t step = 32;
    // the answer lies in [lo, hi]; hi itself when every entry below it is < key
    while (hi - lo > 32) {
        const int64_t idx = (int64_t)lo + (int64_t)(lane + 1) * step - 1;
        const bool lt = idx < hi && (GLOBAL ? __ldg(a + idx) : a[idx]) < key;
        const int cnt = __popc(__ballot_sync(FULL, lt));
        if (cnt == 32) {
            lo = (int32_t)min((int64_t)hi, (int64_t)lo + 32 * step);
        } else {
            lo = (int32_t)((int64_t)lo + cnt * step);
            hi = (int32_t)min((int64_t)hi, (int64_t)lo + step - 1);
        }
        step = ((int64_t)(hi - lo) + 31) >> 5;
    }
    const bool lt = lo + lane < hi && (GLOBAL ? __ldg(a + lo + lane) : a[lo + lane]) < key;
    return lo + __popc(__ballot_sync(FULL, lt));
}

// Warp-cooperative sorted merge of B row [bs, be) against the item's sorted
// mask columns; matches add a*b into the slot accumulator. Each step ranks
// 32 B entries against 32 mask columns; the side whose run ends first moves
// past what it resolved, and when the entry 64 ahead on that side is still
// below the other side's first unresolved value, it gallops there by a warp
// search instead of walking (a hub B row against a short mask row costs a
// few searches per mask column, not a pass over the hub). Returns the B
// entries it compared.
template <typename T, typename A>
__device__ __forceinline__ int32_t merge_row(const MxmArgs<T, A>& p, int32_t bs, int32_t be, A av,
                                             const SlotView& v, A* acc) {
    const int lane = threadIdx.x & 31;
    const unsigned FULL = 0xffffffffu;
    if (bs >= be) return 0;
    int32_t yc = warp_lower_bound<false>(v.mcol, 0, v.ns, __ldg(p.bc + bs));
    int32_t xb = bs, seen = 0;
    while (xb < be && yc < v.ns) {
        const int32_t x = (xb + lane < be) ? __ldg(p.bc + xb + lane) : INT32_MAX;
        const int32_t xp = (xb + 63 < be) ? __ldg(p.bc + xb + 63) : INT32_MAX;  // end of the next B run
        const int32_t y = (yc + lane < v.ns) ? v.mcol[yc + lane] : INT32_MAX;
        const int32_t yp = (yc + 63 < v.ns) ? v.mcol[yc + 63] : INT32_MAX;  // end of the next mask run
        seen += min(32, be - xb);
        int r = 0;
#pragma unroll
        for (int step = 16; step >= 1; step >>= 1) {
            const int32_t yy = __shfl_sync(FULL, y, r + step - 1);
            if (yy < x) r += step;
        }
        const int32_t y31 = __shfl_sync(FULL, y, 31);
        if (r == 31 && y31 < x) r = 32;
        const int32_t yr = __shfl_sync(FULL, y, r & 31);
        if (r < 32 && yr == x && x != INT32_MAX)
            atomic_add_acc<A>(&acc[yc + r], av * to_acc<T, A>(__ldg(p.bv + xb + lane)));
        // the run whose last element is smaller is resolved; for B that is
        // its last stored element (past the row's end the lanes hold INT32_MAX)
        const int32_t xl = __shfl_sync(FULL, x, min(31, be - 1 - xb));
        if (xl <= y31) {
            // mask columns <= xl are resolved too; yu: the first one above
            const unsigned gt = __ballot_sync(FULL, y > xl);
            if (gt == 0u) {
                xb += 32;
                yc += 32;
            } else {
                const int f = __ffs(gt) - 1;
                const int32_t yu = __shfl_sync(FULL, y, f);
                yc += f;
                xb = xp < yu ? warp_lower_bound<true>(p.bc, xb + 64, be, yu) : xb + 32;
            }
        } else {
            // B entries <= y31 are resolved; xu: the first one above
            const int g = __ffs(__ballot_sync(FULL, x > y31)) - 1;
            const int32_t xu = __shfl_sync(FULL, x, g);
            xb += g;
            yc = yp < xu ? warp_lower_bound<false>(v.mcol, yc + 64, v.ns, xu) : yc + 32;
        }
    }
    return seen;
}

// One lane's sorted merge of B row [bs, be) against the mask columns: a
// binary search places the first B column, then the mask position gallops
// (doubling steps, then a binary search) to the first column >= each next
// B column. B columns are loaded four at a time, the next four while the
// current ones are merged.
template <typename T, typename A>
__device__ __forceinline__ void lane_merge(const MxmArgs<T, A>& p, int32_t bs, int32_t be, A av, const SlotView& v,
                                           A* acc) {
    const int32_t* mc = v.mcol;
    const int32_t ns = v.ns;
    int32_t xn[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) xn[q] = bs + q < be ? __ldg(p.bc + bs + q) : INT32_MAX;
    int32_t yc = lower_bound_i32(mc, ns, xn[0]);
    if (yc >= ns) return;
    for (int32_t j = bs; j < be; j += 4) {
        int32_t x[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            x[q] = xn[q];
            xn[q] = j + 4 + q < be ? __ldg(p.bc + j + 4 + q) : INT32_MAX;
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            if (j + q >= be) break;
            if (mc[yc] < x[q]) {
                int32_t b = 1;
                while (yc + b < ns && mc[yc + b] < x[q]) b <<= 1;
                // mc[yc + b/2] < x; mc[yc + b] >= x unless past the end
                int32_t lo = yc + (b >> 1) + 1, hi = min(ns, yc + b);
                while (lo < hi) {
                    const int32_t mid = (lo + hi) >> 1;
                    if (mc[mid] < x[q]) lo = mid + 1; else hi = mid;
                }
                yc = lo;
                if (yc >= ns) return;
            }
            if (mc[yc] == x[q]) atomic_add_acc<A>(&acc[yc], av * to_acc<T, A>(__ldg(p.bv + j + q)));
        }
    }
}

// The lane's share of B entries [j0, j1) cut into 32 contiguous slices,
// merged against the mask by one lane each.
template <typename T, typename A>
__device__ __forceinline__ void merge_slices(const MxmArgs<T, A>& p, int32_t j0, int32_t j1, A av, const SlotView& v,
                                             A* acc) {
    const int32_t per = (j1 - j0 + 31) >> 5;
    const int32_t s0 = j0 + (threadIdx.x & 31) * per, s1 = min(j1, s0 + per);
    if (s0 < s1) lane_merge<T, A>(p, s0, s1, av, v, acc);
}

// Merge variant, 32 A entries at a time (lane l takes entry t0 + l). A B
// row whose part inside [lo, hi] has at most kLaneMerge entries is merged by
// its own lane. In a CTA item (PUSH) one with more than kMergePiece entries
// is listed for the CTA, which cuts it into pieces that all warps share.
// The others are merged by the whole warp afterwards, one at a time: cut
// into 32 slices (merge_slices); or, when a B row is more than kMergeRatio
// times longer than the mask row, by the warp-cooperative merge (which
// gallops over the long B row). Returns the B entries compared
// (warp-uniform; listed rows are counted where their pieces are merged).
constexpr int kLaneMerge = 8;
constexpr int kMergeRatio = 8;
constexpr int kMergePiece = 256;
template <typename T, typename A, bool PUSH>
__device__ __forceinline__ int64_t merge_group(const MxmArgs<T, A>& p, int32_t t0, int32_t ae, bool clip,
                                               const SlotView& v, A* acc, int* s_nlong, int32_t* s_lbs,
                                               int32_t* s_lend, A* s_la) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int32_t t = t0 + lane;
    int32_t bs = 0, be = 0;
    A av = (A)0;
    if (t < ae) {
        b_range(p, t, clip, v.lo, v.hi, bs, be);
        av = to_acc<T, A>(__ldg(p.av + t));
        if (PUSH && be - bs > kMergePiece) {
            const int slot = atomicAdd(s_nlong, 1);
            if (slot < kLongCap) {
                s_lbs[slot] = bs;
                s_lend[slot] = be;
                s_la[slot] = av;
                be = bs;
            }
        }
    }
    const bool wide = be - bs > kLaneMerge;
    if (!wide && bs < be) lane_merge<T, A>(p, bs, be, av, v, acc);
    int64_t seen = warp_sum<int64_t>(wide ? 0 : be - bs);
    for (unsigned w = __ballot_sync(FULL, wide); w; w &= w - 1) {
        const int l = __ffs(w) - 1;
        const int32_t s = __shfl_sync(FULL, bs, l), e = __shfl_sync(FULL, be, l);
        const A a = __shfl_sync(FULL, av, l);
        if ((int64_t)v.ns * kMergeRatio < (int64_t)(e - s)) {
            seen += merge_row<T, A>(p, s, e, a, v, acc);
        } else {
            merge_slices<T, A>(p, s, e, a, v, acc);
            seen += e - s;
        }
    }
    return seen;
}

// Shared-memory layout per variant (MD of the CTA phase: MD_DENSE for MSA).
template <int MD, typename A, bool SLOTS>
struct MxmSmem {
    static constexpr bool dense = MD == MD_DENSE;
    // CTA phase
    static constexpr size_t off_acc = 0;
    static constexpr size_t off_lbs = off_acc + (size_t)kCtaSlots<A> * sizeof(A);
    static constexpr size_t off_lend = off_lbs + (size_t)kLongCap * 4;
    static constexpr size_t off_lchunk = off_lend + (size_t)kLongCap * 4;
    static constexpr size_t off_la = off_lchunk + (size_t)(kLongCap + 8) * 4;
    static constexpr size_t off_key = off_la + (size_t)kLongCap * sizeof(A);  // bits and wbase, or mcol
    static constexpr size_t off_wbase = off_key + (size_t)kWinWords * 4 + 16;  // behind a guard word
    static constexpr size_t cta_bytes =
        dense ? off_wbase + (size_t)kWinWords * 2 : off_key + (size_t)kCtaSlots<A> * 4;
    // warp phase (per warp): acc and mcol; or acc, hkeys, hslot and the filter;
    // or, by slots, acc and mcol over the first two, hslot, the filter and used
    static constexpr size_t w_acc = 0;
    static constexpr size_t w_mcol = w_acc + (size_t)kWarpSlots * sizeof(A);
    static constexpr size_t w_hkeys = w_acc + (size_t)kColumnSlots<A> * sizeof(A);
    static constexpr size_t w_hslot = w_hkeys + (size_t)(1 << kWarpTblBits) * 4;
    static constexpr size_t w_filt = w_hslot + (size_t)(1 << kWarpTblBits);
    static constexpr size_t w_used = w_filt + (size_t)(1 << kFilterBits) / 8;
    static constexpr size_t warp_one = !dense ? w_mcol + (size_t)kWarpSlots * 4
                                       : SLOTS ? w_used + (size_t)(1 << kWarpTblBits) / 8
                                               : w_used;
    static_assert(!SLOTS || w_mcol + (size_t)kWarpSlots * 4 <= w_hslot, "acc and mcol end before the table of slots");
    static constexpr size_t warp_bytes = warp_one * kMxmWarps;
    static constexpr size_t region = cta_bytes > warp_bytes ? cta_bytes : warp_bytes;
    // per-warp flattening scratch (both phases)
    static constexpr size_t scratch_bytes = (size_t)kMxmWarps * 32 * (2 * sizeof(int) + sizeof(A));
    static constexpr size_t total = region + scratch_bytes;
};

template <int MD, int VM, typename T, typename A, bool SLOTS>
__global__ void __launch_bounds__(kMxmThreads, 3) k_mxm_masked(MxmArgs<T, A> p) {
    extern __shared__ __align__(16) unsigned char smem[];
    using SM = MxmSmem<MD, A, SLOTS>;
    constexpr bool DENSE = MD == MD_DENSE;
    constexpr int WMD = DENSE ? MD_HASHED : MD;  // warp-row lookup
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    unsigned char* scr = smem + SM::region;
    int* s_incl = reinterpret_cast<int*>(scr) + wid * 32;
    int* s_off = reinterpret_cast<int*>(scr) + kMxmWarps * 32 + wid * 32;
    A* s_a = reinterpret_cast<A*>(scr + (size_t)kMxmWarps * 32 * 2 * sizeof(int)) + wid * 32;
    __shared__ int s_item, s_nlong, s_nchunks, s_chunk_next;
    unsigned long long executed = 0;  // products this warp processed (warp-uniform)

    // ------------------------------------------------------------ CTA items
    const int nheavy = p.q->heavy_count;
    const int ncta = nheavy + p.q->normal_count;
    if (ncta) {
        A* acc = reinterpret_cast<A*>(smem + SM::off_acc);
        int32_t* lbs = reinterpret_cast<int32_t*>(smem + SM::off_lbs);
        int32_t* lend = reinterpret_cast<int32_t*>(smem + SM::off_lend);
        int32_t* lchunk = reinterpret_cast<int32_t*>(smem + SM::off_lchunk);
        A* la = reinterpret_cast<A*>(smem + SM::off_la);
        uint32_t* bits = reinterpret_cast<uint32_t*>(smem + SM::off_key);
        uint16_t* wbase = reinterpret_cast<uint16_t*>(smem + SM::off_wbase);
        int32_t* mcol = reinterpret_cast<int32_t*>(smem + SM::off_key);
        if (DENSE)
            for (int t = threadIdx.x; t <= kWinWords; t += blockDim.x) bits[t] = 0u;
        while (true) {
            if (threadIdx.x == 0) {
                s_item = atomicAdd(&p.q->cta_next, 1);
                s_nlong = 0;
            }
            __syncthreads();
            const int it = s_item;
            if (it >= ncta) break;
            const int4 item = p.cta_items[it < nheavy ? it : p.cta_cap - 1 - (it - nheavy)];
            const int64_t i = item.x;
            const int32_t mb = p.mr[i], mi = p.mre[i] - mb;
            const int s0 = item.y, ns = item.z - item.y;
            const int32_t* gcol = p.mc + mb + s0;
            SlotView v;
            v.mcol = mcol; v.bits = bits; v.wbase = wbase; v.filt = nullptr; v.hkeys = nullptr; v.hslot = nullptr;
            v.ns = ns;
            v.lo = __ldg(gcol); v.hi = __ldg(gcol + ns - 1);
            for (int s = threadIdx.x; s < ns; s += blockDim.x) {
                const int32_t c = __ldg(gcol + s);
                acc[s] = (A)0;
                if (DENSE) {
                    const uint32_t d = (uint32_t)(c - v.lo);
                    atomicOr(&bits[d >> 5], 1u << (d & 31));
                    if (s == 0 || ((uint32_t)(__ldg(gcol + s - 1) - v.lo) >> 5) != (d >> 5)) wbase[d >> 5] = (uint16_t)s;
                } else {
                    mcol[s] = c;
                }
            }
            __syncthreads();
            // a window that does not span the whole row, or a mask restricted
            // to part of the row, only meets B entries inside [lo, hi]
            const bool clip = ns < mi || p.clip;
            const int32_t ab = p.ar[i], ae = p.are[i];
            if (MD == MD_MERGE) {
                // phase A: groups of up to 32 A entries, small enough that
                // every warp gets one when the row is short; B rows longer
                // than kMergePiece listed
                const int32_t gsz = min(32, (ae - ab + kMxmWarps - 1) / kMxmWarps);
                for (int32_t g = ab + wid * gsz; g < ae; g += kMxmWarps * gsz)
                    executed += (unsigned long long)merge_group<T, A, true>(p, g, min(ae, g + gsz), clip, v, acc,
                                                                            &s_nlong, lbs, lend, la);
            } else {
                // phase A: short B rows flattened per warp, long ones listed
                // (an A row too short to give every warp 32 entries lists
                // its B rows from 32 entries up, so all warps share them)
                const int long_seg = ae - ab < kShortARow ? kLongSegShort : kLongSeg;
                for (int32_t g = ab + wid * 32; g < ae; g += kMxmWarps * 32)
                    executed += (unsigned long long)group_products<MD, VM, T, A, true>(
                        p, g, ae, clip, v, acc, s_incl, s_off, s_a, &s_nlong, lbs, lend, la, long_seg);
            }
            __syncthreads();
            {
                // phase B: long B rows cut into kChunk pieces shared by all warps
                const int nlong = min(s_nlong, kLongCap);
                if (nlong > 0) {
                    if (wid == 0) {
                        int running = 0;
                        for (int base = 0; base < nlong; base += 32) {
                            const int x = base + lane;
                            const int c = x < nlong ? (lend[x] - lbs[x] + kChunk - 1) / kChunk : 0;
                            const int incl = warp_incl_scan(c);
                            if (x < nlong) lchunk[x + 1] = running + incl;
                            running += __shfl_sync(FULL, incl, 31);
                        }
                        if (lane == 0) {
                            lchunk[0] = 0;
                            s_nchunks = running;
                            s_chunk_next = 0;
                        }
                    }
                    __syncthreads();
                    const int nch = s_nchunks;
                    while (true) {
                        int c = 0;
                        if (lane == 0) c = atomicAdd(&s_chunk_next, 1);
                        c = __shfl_sync(FULL, c, 0);
                        if (c >= nch) break;
                        const int seg = upper_bound_i32(lchunk + 1, nlong, c);
                        const int32_t j0 = lbs[seg] + (c - lchunk[seg]) * kChunk;
                        const int32_t j1 = min(lend[seg], j0 + kChunk);
                        if (MD == MD_MERGE) merge_slices<T, A>(p, j0, j1, la[seg], v, acc);
                        else stream_row<MD, VM, T, A>(p, v, acc, j0, j1, la[seg]);
                        executed += (unsigned long long)(j1 - j0);
                    }
                }
            }
            __syncthreads();
            for (int s = threadIdx.x; s < ns; s += blockDim.x) {
                p.cv[mb + s0 + s] = from_acc<T, A>(acc[s]);
                if (DENSE) bits[(uint32_t)(__ldg(gcol + s) - v.lo) >> 5] = 0u;
            }
            __syncthreads();
        }
    }

    // ----------------------------------------------------------- warp rows
    {
        unsigned char* base = smem + wid * SM::warp_one;
        A* acc = reinterpret_cast<A*>(base + SM::w_acc);
        uint32_t* filt = reinterpret_cast<uint32_t*>(base + SM::w_filt);
        int32_t* hkeys = reinterpret_cast<int32_t*>(base + SM::w_hkeys);
        uint8_t* hslot = reinterpret_cast<uint8_t*>(base + SM::w_hslot);
        int32_t* mcol = reinterpret_cast<int32_t*>(base + SM::w_mcol);
        uint32_t* used = reinterpret_cast<uint32_t*>(base + SM::w_used);
        constexpr int FW = (1 << kFilterBits) / 32;
        constexpr int TBL = 1 << kWarpTblBits;
        if (DENSE)
            for (int t = lane; t < FW; t += 32) filt[t] = 0u;
        if (DENSE)
            for (int t = lane; t < TBL; t += 32) hkeys[t] = kEmpty;
        __syncwarp();
        // Without CTA items every warp's first row is its own number: all
        // 7,296 warps taking a row from the counter, most to find none, are
        // half the time of a small product (1,000 rows: 9.9 us, so 6.3; 4,786 rows 44 and 36).
        const int nwarp = p.q->warp_count, dealt = ncta ? 0 : gridDim.x * kMxmWarps;
        for (bool first = ncta == 0;; first = false) {
            int r = blockIdx.x + wid * gridDim.x;
            if (!first) {
                if (lane == 0) r = dealt + atomicAdd(&p.q->warp_next, 1);
                r = __shfl_sync(FULL, r, 0);
            }
            if (r >= nwarp) break;
            const int64_t i = p.warp_rows[r];
            const int32_t mb = p.mr[i], mi = p.mre[i] - mb;
            const bool clip = p.clip;
            const int32_t* gcol = p.mc + mb;
            SlotView v;
            v.mcol = mcol; v.bits = nullptr; v.wbase = nullptr; v.filt = filt; v.hkeys = hkeys; v.hslot = hslot;
            v.ns = mi;
            v.lo = __ldg(gcol); v.hi = __ldg(gcol + mi - 1);
            const bool by_slots = SLOTS && mi > kColumnSlots<A>;
            if (by_slots) {
                if (lane < TBL / 32) used[lane] = 0u;
                for (int t = lane; t < TBL / 4; t += 32) reinterpret_cast<uint32_t*>(hslot)[t] = ~0u;
                __syncwarp();
            }
            for (int s = lane; s < mi; s += 32) {
                const int32_t c = __ldg(gcol + s);
                acc[s] = (A)0;
                if (DENSE) {
                    const uint32_t h = hash_col(c);
                    const uint32_t f = h >> (32 - kFilterBits);
                    atomicOr(&filt[f >> 5], 1u << (f & 31));
                }
                if (by_slots) {
                    mcol[s] = c;
                    if (s + 1 < mi) slot_insert(used, hslot, c, s);
                } else if (DENSE) {
                    hash_insert<uint8_t>(hkeys, hslot, kWarpTblBits, c, (uint8_t)s);
                } else {
                    mcol[s] = c;
                }
            }
            __syncwarp();
            const int32_t ab = p.ar[i], ae = p.are[i];
            if (MD == MD_MERGE) {
                for (int32_t g = ab; g < ae; g += 32)
                    executed += (unsigned long long)merge_group<T, A, false>(p, g, ae, clip, v, acc, nullptr,
                                                                             nullptr, nullptr, nullptr);
            } else if (by_slots) {
                for (int32_t g = ab; g < ae; g += 32)
                    executed += (unsigned long long)group_products<SLOTS ? MD_SLOTS : WMD, VM, T, A, false>(
                        p, g, ae, clip, v, acc, s_incl, s_off, s_a, nullptr, nullptr, nullptr, nullptr);
            } else {
                for (int32_t g = ab; g < ae; g += 32)
                    executed += (unsigned long long)group_products<WMD, VM, T, A, false>(
                        p, g, ae, clip, v, acc, s_incl, s_off, s_a, nullptr, nullptr, nullptr, nullptr);
            }
            __syncwarp();
            for (int s = lane; s < mi; s += 32) p.cv[mb + s] = from_acc<T, A>(acc[s]);
            if (by_slots) __syncwarp();  // the table of columns lies over acc
            if (DENSE)
                for (int t = lane; t < FW; t += 32) filt[t] = 0u;
            if (DENSE)
                for (int t = lane; t < TBL; t += 32) hkeys[t] = kEmpty;
            __syncwarp();
        }
    }
    if (lane == 0 && executed) atomicAdd(&p.ctr[GA_CTR_EXECUTED], executed);
}

static int64_t cta_item_cap(int64_t m, int64_t n, int64_t mask_nnz) {
    // windows per row <= ceil(m_i / kLeastCtaSlots) + ceil(n / kWinCols), and <= m_i;
    // kSplitItems for the split rows
    const int64_t per_row = 1 + (n + kWinCols - 1) / kWinCols;
    int64_t cap = m * per_row + mask_nnz / kLeastCtaSlots + 1 + kSplitItems;
    if (cap > mask_nnz + 1) cap = mask_nnz + 1;
    return cap;
}

// Launch the masked product for one value type and lookup variant.
template <int LK, int VM, typename T>
static void launch_masked(ga_ctx ctx, ga_csr A_, ga_csr B_, ga_csr M_, T* cv, MxmQueue* q, int32_t* warp_rows,
                          int4* cta_items, int32_t cta_cap, const int32_t* mre, const MxmRows& rows, const char* name,
                          const int32_t* btr = nullptr, int2* dot_tasks = nullptr) {
    using Ac = typename Acc<T>::type;
    MxmArgs<T, Ac> p;
    p.ar = A_->rst; p.ac = A_->col; p.av = static_cast<const T*>(A_->val);
    p.br = B_->rst; p.bc = B_->col; p.bv = static_cast<const T*>(B_->val);
    p.mr = M_->rst; p.mc = M_->col;
    p.are = rows.a_end ? rows.a_end : A_->rst + 1;
    p.bre = rows.b_end ? rows.b_end : B_->rst + 1;
    p.mre = mre ? mre : M_->rst + 1;
    p.cmr = rows.counted ? rows.counted : p.mr;
    p.cme = rows.counted ? rows.counted + 1 : p.mre;
    p.clip = mre != nullptr && rows.clip;
    p.cv = cv; p.m = M_->m; p.q = q; p.warp_rows = warp_rows; p.cta_items = cta_items; p.cta_cap = cta_cap;
    p.ctr = ctx->d_counters;
    p.heavy_flops = ctx->tune.heavy_flops;
    p.split = LK == MD_MERGE ? kSplitMerge : kSplit;
    constexpr bool kHasSlots = LK == MD_DENSE && kColumnSlots<Ac> < kWarpSlots;
    const bool slots = kHasSlots && M_->nnz > (int64_t)kSlotsMean * p.m;
    const bool all = LK == MD_MERGE ? p.m > (int64_t)kFewRows * ctx->num_sms : slots;
    p.warp_slots = all ? kWarpSlots : kColumnSlots<Ac>;
    p.warp_max_flops = ctx->tune.warp_max_flops;
    // the limit reaches the option's default at (32,768 / kWarpShare)^2
    // products; rows of mean length give a lower bound of their number
    const double most = (double)MxmTune().warp_max_flops / kWarpShare;
    p.small = p.m > 0 && (double)A_->nnz * (double)B_->nnz < most * most * (double)B_->m;
    p.btr = btr;
    p.dot_tasks = dot_tasks;
    p.hybrid_ratio = ctx->tune.hybrid_ratio;
    {
        ProfScope ps(ctx, "mxm_row_bin");
        const int take = (int)std::min<int64_t>(32, std::max<int64_t>(1, p.m / (ctx->num_sms * 64)));
        const int grid = grid_for((p.m + take - 1) / take * 32, kBinThreads, ctx->num_sms * 16);
        k_row_bin<T, Ac><<<grid, kBinThreads, 0, ctx->stream>>>(p, take);
        post_launch("mxm_row_bin");
    }
    const size_t smem = slots ? MxmSmem<LK, Ac, kHasSlots>::total : MxmSmem<LK, Ac, false>::total;
    auto kern = slots ? k_mxm_masked<LK, VM, T, Ac, kHasSlots> : k_mxm_masked<LK, VM, T, Ac, false>;
    GA_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    int per_sm = 0;
    GA_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, kMxmThreads, smem));
    if (per_sm < 1) per_sm = 1;
    if (ctx->tune.ctas_per_sm > 0 && ctx->tune.ctas_per_sm < per_sm) per_sm = ctx->tune.ctas_per_sm;
    ProfScope ps(ctx, name);
    kern<<<ctx->num_sms * per_sm, kMxmThreads, smem, ctx->stream>>>(p);
    post_launch(name);
}

// ------------------------------------------------------- inner-product form
// C<M>(i, j) = sum over k in A_i ∩ (B^T)_j of A(i, k) * B(k, j): one warp per
// mask entry, the shorter of the two sorted lists walked 32 entries at a
// time (one per lane), each lane binary-searching the longer one. Warps take
// `chunk` consecutive mask entries; a chunk finds its row by a binary
// search of the row partition `seg`. Row i's mask is [lo[i], hi[i]) within
// the partition [seg[i], seg[i+1]) (the k-truss support evaluates only the
// upper part of each row). No shared memory and no atomics: each mask entry
// is written by one warp.
constexpr int kDotThreads = 256;

template <typename T>
struct DotArgs {
    const int32_t* ar; const int32_t* ac; const T* av;
    const int32_t* tr; const int32_t* tc; const T* tv;  // B^T
    const int32_t* br;                                  // B row starts (product count)
    const int32_t* seg; const int32_t* lo; const int32_t* hi;
    const int32_t* cmr; const int32_t* cme;             // mask rows that the work counters count
    const int32_t* mc;
    T* cv;
    int64_t m, total;
    int chunk;  // mask entries per warp task
    unsigned long long* ctr;
};

// Gustavson products of the masked rows (the work every other variant does),
// mask entries and launch counters, as k_row_bin counts them.
template <typename T>
__global__ void k_dot_count(DotArgs<T> p) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    unsigned long long my_flops = 0, my_mask = 0;
    if (blockIdx.x == 0 && threadIdx.x == 0) {
        atomicAdd(&p.ctr[GA_CTR_LAUNCHES], 1ull);
        atomicAdd(&p.ctr[GA_CTR_A_ENTRIES], (unsigned long long)(p.ar[p.m] - p.ar[0]));
        atomicAdd(&p.ctr[GA_CTR_ROWS], (unsigned long long)p.m);
    }
    for (int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; i < p.m; i += warps) {
        const int32_t mi = p.cme[i] - p.cmr[i];
        if (mi <= 0) continue;
        long long f = 0;
        for (int32_t t = p.ar[i] + lane; t < p.ar[i + 1]; t += 32) {
            const int32_t k = p.ac[t];
            f += p.br[k + 1] - p.br[k];
        }
        f = warp_sum<long long>(f);
        if (lane == 0) {
            my_flops += (unsigned long long)f;
            my_mask += (unsigned long long)mi;
        }
    }
    if (lane == 0 && my_flops) atomicAdd(&p.ctr[GA_CTR_PRODUCTS], my_flops);
    if (lane == 0 && my_mask) atomicAdd(&p.ctr[GA_CTR_MASK_ENTRIES], my_mask);
}

template <typename T, bool UNIT>
__global__ void __launch_bounds__(kDotThreads) k_mxm_dot(DotArgs<T> p) {
    using Ac = typename Acc<T>::type;
    const int lane = threadIdx.x & 31;
    const unsigned FULL = 0xffffffffu;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    unsigned long long executed = 0;
    // entries of the partition as the device holds it now (inside a captured
    // k-truss loop, p.total is only the launch-time upper bound)
    const int64_t total = p.seg[p.m];
    for (int64_t c = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; c * p.chunk < total; c += warps) {
        const int32_t q0 = (int32_t)(c * p.chunk);
        const int32_t q1 = (int32_t)min((int64_t)q0 + p.chunk, total);
        int i = upper_bound_i32(p.seg, (int)p.m + 1, q0) - 1;
        for (int32_t q = q0; q < q1; ++q) {
            while (q >= p.seg[i + 1]) ++i;
            if (q < p.lo[i] || q >= p.hi[i]) continue;
            const int32_t j = p.mc[q];
            const int32_t ab = p.ar[i], an = p.ar[i + 1] - ab;
            const int32_t tb = p.tr[j], tn = p.tr[j + 1] - tb;
            Ac s = 0;
            if (an > 0 && tn > 0) {
                const bool walk_a = an <= tn;  // walk the shorter list, search the longer
                const int32_t* Wc = walk_a ? p.ac + ab : p.tc + tb;
                const int32_t* Sc = walk_a ? p.tc + tb : p.ac + ab;
                const int wn = walk_a ? an : tn, sn = walk_a ? tn : an;
                if (lane == 0) executed += (unsigned long long)wn;
                // The searched list in registers: up to 32 entries one per
                // lane (searched by shuffles, no memory access), else, when
                // 32 or more entries are walked, the last entry of each of 32
                // equal buckets (the shuffle search picks the bucket, a
                // binary search in memory finishes); else a plain binary
                // search.
                // bucket splitters pay off only when at least 32 entries are walked
                const bool small = sn <= 32, bucketed = !small && wn >= 32;
                int32_t key = INT32_MAX;
                if (small) {
                    key = lane < sn ? __ldg(Sc + lane) : INT32_MAX;
                } else if (bucketed) {
                    const int hi_b = (int)(((int64_t)(lane + 1) * sn) >> 5);
                    key = __ldg(Sc + hi_b - 1);
                }
                for (int base = 0; base < wn; base += 32) {
                    const int e = base + lane;
                    const int32_t x = e < wn ? __ldg(Wc + e) : INT32_MAX;
                    // first register entry >= x (32: none)
                    const int b = (small || bucketed) ? warp_lower_bound(key, x) : 0;
                    bool hit = false;
                    int pos = 0;
                    if (small) {
                        const int32_t y = __shfl_sync(FULL, key, b & 31);
                        pos = b;
                        hit = e < wn && b < sn && y == x;
                    } else if (bucketed) {
                        if (e < wn && b < 32) {
                            const int lo_b = (int)(((int64_t)b * sn) >> 5);
                            const int hi_b = (int)(((int64_t)(b + 1) * sn) >> 5);
                            pos = lo_b + lower_bound_i32(Sc + lo_b, hi_b - lo_b, x);
                            hit = pos < hi_b && __ldg(Sc + pos) == x;
                        }
                    } else if (e < wn) {
                        pos = lower_bound_i32(Sc, sn, x);
                        hit = pos < sn && __ldg(Sc + pos) == x;
                    }
                    if (UNIT) {
                        s += (Ac)__popc(__ballot_sync(FULL, hit));
                    } else if (hit) {
                        const T va = walk_a ? p.av[ab + e] : p.av[ab + pos];
                        const T vb = walk_a ? p.tv[tb + pos] : p.tv[tb + e];
                        s += (Ac)va * (Ac)vb;
                    }
                }
                if (!UNIT) s = warp_sum<Ac>(s);
            }
            if (lane == 0) p.cv[q] = (T)s;
        }
    }
    if (lane == 0 && executed) atomicAdd(&p.ctr[GA_CTR_EXECUTED_DOT], executed);
}

// Hybrid form, inner-product rows: one warp per listed task (a row and up
// to kDotTask of its mask entries), each entry an intersection as in k_mxm_dot.
template <typename T, bool UNIT>
__global__ void __launch_bounds__(kDotThreads) k_mxm_dot_rows(DotArgs<T> p, const int2* __restrict__ tasks,
                                                              const MxmQueue* __restrict__ q) {
    using Ac = typename Acc<T>::type;
    const int lane = threadIdx.x & 31;
    const unsigned FULL = 0xffffffffu;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    const int n = q->dot_count;
    unsigned long long executed = 0;
    for (int64_t r = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5; r < n; r += warps) {
        const int2 task = tasks[r];
        const int32_t i = task.x;
        const int32_t ab = p.ar[i], an = p.ar[i + 1] - ab;
        const int32_t q_end = min(p.hi[i], task.y + kDotTask);
        for (int32_t qq = task.y; qq < q_end; ++qq) {
            const int32_t j = p.mc[qq];
            const int32_t tb = p.tr[j], tn = p.tr[j + 1] - tb;
            Ac s = 0;
            if (an > 0 && tn > 0) {
                const bool walk_a = an <= tn;
                const int32_t* Wc = walk_a ? p.ac + ab : p.tc + tb;
                const int32_t* Sc = walk_a ? p.tc + tb : p.ac + ab;
                const int wn = walk_a ? an : tn, sn = walk_a ? tn : an;
                if (lane == 0) executed += (unsigned long long)wn;
                const bool small = sn <= 32, bucketed = !small && wn >= 32;
                int32_t key = INT32_MAX;
                if (small) {
                    key = lane < sn ? __ldg(Sc + lane) : INT32_MAX;
                } else if (bucketed) {
                    const int hi_b = (int)(((int64_t)(lane + 1) * sn) >> 5);
                    key = __ldg(Sc + hi_b - 1);
                }
                for (int base = 0; base < wn; base += 32) {
                    const int e = base + lane;
                    const int32_t x = e < wn ? __ldg(Wc + e) : INT32_MAX;
                    const int b = (small || bucketed) ? warp_lower_bound(key, x) : 0;
                    bool hit = false;
                    int pos = 0;
                    if (small) {
                        const int32_t y = __shfl_sync(FULL, key, b & 31);
                        pos = b;
                        hit = e < wn && b < sn && y == x;
                    } else if (bucketed) {
                        if (e < wn && b < 32) {
                            const int lo_b = (int)(((int64_t)b * sn) >> 5);
                            const int hi_b = (int)(((int64_t)(b + 1) * sn) >> 5);
                            pos = lo_b + lower_bound_i32(Sc + lo_b, hi_b - lo_b, x);
                            hit = pos < hi_b && __ldg(Sc + pos) == x;
                        }
                    } else if (e < wn) {
                        pos = lower_bound_i32(Sc, sn, x);
                        hit = pos < sn && __ldg(Sc + pos) == x;
                    }
                    if (UNIT) {
                        s += (Ac)__popc(__ballot_sync(FULL, hit));
                    } else if (hit) {
                        const T va = walk_a ? p.av[ab + e] : p.av[ab + pos];
                        const T vb = walk_a ? p.tv[tb + pos] : p.tv[tb + e];
                        s += (Ac)va * (Ac)vb;
                    }
                }
                if (!UNIT) s = warp_sum<Ac>(s);
            }
            if (lane == 0) p.cv[qq] = (T)s;
        }
    }
    if (lane == 0 && executed) atomicAdd(&p.ctr[GA_CTR_EXECUTED_DOT], executed);
}

template <typename T>
static void launch_dot_t(ga_ctx ctx, ga_csr A, ga_csr B, ga_csr Bt, ga_csr M, T* cv, bool unit,
                         const int32_t* mre, const int32_t* counted, const int2* dot_tasks = nullptr,
                         const MxmQueue* q = nullptr) {
    DotArgs<T> p;
    p.ar = A->rst; p.ac = A->col; p.av = static_cast<const T*>(A->val);
    p.tr = Bt->rst; p.tc = Bt->col; p.tv = static_cast<const T*>(Bt->val);
    p.br = B->rst;
    // with mask row ends, M's columns are those of the CSR whose row starts
    // are mre - 1 (the partition of the entries); else M's own rows
    p.seg = mre ? mre - 1 : M->rst;
    p.lo = M->rst;
    p.hi = mre ? mre : M->rst + 1;
    p.cmr = counted ? counted : p.lo;
    p.cme = counted ? counted + 1 : p.hi;
    p.mc = M->col;
    p.cv = cv; p.m = M->m; p.ctr = ctx->d_counters;
    p.total = M->nnz;
    p.chunk = ctx->tune.dot_chunk > 0 ? ctx->tune.dot_chunk : 8;
    if (dot_tasks) {  // hybrid form: the tasks binning listed (it also counted the work)
        ProfScope ps(ctx, "mxm_dot_rows");
        const int grid = ctx->num_sms * (2048 / kDotThreads);
        if (unit) k_mxm_dot_rows<T, true><<<grid, kDotThreads, 0, ctx->stream>>>(p, dot_tasks, q);
        else k_mxm_dot_rows<T, false><<<grid, kDotThreads, 0, ctx->stream>>>(p, dot_tasks, q);
        post_launch("mxm_dot_rows");
        return;
    }
    {
        ProfScope ps(ctx, "mxm_dot_count");
        k_dot_count<T><<<grid_for(p.m * 32, 256, ctx->num_sms * 16), 256, 0, ctx->stream>>>(p);
        post_launch("mxm_dot_count");
    }
    if (p.total == 0) return;
    const int grid = grid_for((p.total + p.chunk - 1) / p.chunk * 32, kDotThreads, ctx->num_sms * 16);
    ProfScope ps(ctx, "mxm_dot");
    if (unit) k_mxm_dot<T, true><<<grid, kDotThreads, 0, ctx->stream>>>(p);
    else k_mxm_dot<T, false><<<grid, kDotThreads, 0, ctx->stream>>>(p);
    post_launch("mxm_dot");
}

// Inner-product launch: Bt holds B^T (B itself when B is symmetric); unit:
// A's and B's values are all ones. Allocates nothing (capturable). With
// mask_row_end, M->nnz must be the entry count of the full partition.
void mxm_dot_launch(ga_ctx ctx, ga_csr A, ga_csr B, ga_csr Bt, ga_csr M, void* d_cvals, bool unit,
                    const int32_t* mask_row_end, const int32_t* counted) {
    GA_DISPATCH_DTYPE(A->dtype, T, {
        launch_dot_t<T>(ctx, A, B, Bt, M, static_cast<T*>(d_cvals), unit, mask_row_end, counted);
    });
}

void naive_masked_into(ga_ctx ctx, ga_csr A, ga_csr B, ga_csr M, void* d_cvals);

// Hybrid form: inner-product tasks, at most one per kDotTask mask entries of a row.
static int64_t dot_task_cap(int64_t m, int64_t mask_nnz) { return mask_nnz / kDotTask + m + 1; }

size_t mxm_scratch_bytes(int64_t m, int64_t n, int64_t mask_nnz, bool hybrid) {
    // queue header, warp rows, CTA items, hybrid inner-product tasks
    return 256 + sizeof(int32_t) * (size_t)(m + 1) + 16 + sizeof(int4) * (size_t)cta_item_cap(m, n, mask_nnz) +
           (hybrid ? sizeof(int2) * (size_t)dot_task_cap(m, mask_nnz) : 0);
}

// Non-allocating launch (usable inside captured loops): `scratch` holds
// mxm_scratch_bytes(M->m, M->n, max nnz(M)) bytes; `cap_nnz` is that max.
// unit_b: B's values are all ones (no value loads). mask_row_end (optional):
// row i's mask is [M->rst[i], mask_row_end[i]) instead of the whole row.
void mxm_masked_launch(ga_ctx ctx, ga_algo algo, ga_csr A, ga_csr B, ga_csr M, void* d_cvals, void* scratch,
                       int64_t cap_nnz, bool unit_b, const int32_t* mask_row_end, bool unit_a, ga_csr Bt,
                       const MxmRows& rows) {
    GA_REQUIRE(algo == GA_MSA || algo == GA_MCA || algo == GA_HEAP || algo == GA_HYBRID, GA_ERR_INVALID_ARG,
               "mxm: unknown algorithm");
    GA_REQUIRE(algo != GA_HYBRID || Bt != nullptr, GA_ERR_INVALID_ARG, "mxm: the hybrid form needs B^T");
    unsigned char* s = static_cast<unsigned char*>(scratch);
    MxmQueue* q = reinterpret_cast<MxmQueue*>(s);
    int32_t* warp_rows = reinterpret_cast<int32_t*>(s + 256);
    size_t off = 256 + sizeof(int32_t) * (size_t)(M->m + 1);
    off = (off + 15) & ~(size_t)15;
    int4* cta_items = reinterpret_cast<int4*>(s + off);
    const int64_t cap = cta_item_cap(M->m, M->n, cap_nnz);
    int2* dot_tasks = algo == GA_HYBRID ? reinterpret_cast<int2*>(s + off + sizeof(int4) * (size_t)cap) : nullptr;
    GA_REQUIRE(cap < INT32_MAX, GA_ERR_UNSUPPORTED, "mxm: too many work items");
    k_reset_queue<<<1, 32, 0, ctx->stream>>>(q);
    post_launch("mxm_reset_queue");
    GA_DISPATCH_DTYPE(A->dtype, T, {
        T* cv = static_cast<T*>(d_cvals);
        const int32_t c32 = (int32_t)cap;
        // value mode 2 (every product is 1) only for int32, the k-truss / TC type
        const bool ones = unit_a && unit_b && std::is_same<T, int32_t>::value;
        if (algo == GA_HYBRID) {
            // Gustavson (MSA) rows, then the inner-product rows flagged while binning
            const int32_t* btr = Bt->rst;
            if (ones)
                launch_masked<MD_DENSE, 2, T>(ctx, A, B, M, cv, q, warp_rows, cta_items, c32, mask_row_end, rows,
                                              "mxm_msa", btr, dot_tasks);
            else if (unit_b)
                launch_masked<MD_DENSE, 1, T>(ctx, A, B, M, cv, q, warp_rows, cta_items, c32, mask_row_end, rows,
                                              "mxm_msa", btr, dot_tasks);
            else
                launch_masked<MD_DENSE, 0, T>(ctx, A, B, M, cv, q, warp_rows, cta_items, c32, mask_row_end, rows,
                                              "mxm_msa", btr, dot_tasks);
            launch_dot_t<T>(ctx, A, B, Bt, M, cv, unit_a && unit_b, mask_row_end, rows.counted, dot_tasks, q);
        } else if (algo == GA_MSA || algo == GA_MCA) {
            const char* name = algo == GA_MSA ? "mxm_msa" : "mxm_mca";
            if (ones)
                launch_masked<MD_DENSE, 2, T>(ctx, A, B, M, cv, q, warp_rows, cta_items, c32, mask_row_end, rows, name);
            else if (unit_b)
                launch_masked<MD_DENSE, 1, T>(ctx, A, B, M, cv, q, warp_rows, cta_items, c32, mask_row_end, rows, name);
            else
                launch_masked<MD_DENSE, 0, T>(ctx, A, B, M, cv, q, warp_rows, cta_items, c32, mask_row_end, rows, name);
        } else {
            launch_masked<MD_MERGE, 0, T>(ctx, A, B, M, cv, q, warp_rows, cta_items, c32, mask_row_end, rows,
                                          "mxm_heap_merge");
        }
    });
}

// C<A> = A·A of a symmetric A: the result is symmetric too, C(j, i) being the
// same products as C(i, j), so half of it is computed. A, B and M are one
// matrix; whether it is symmetric is known to the handle or checked here (a
// search per entry, once per handle, and a synchronisation). From kSymHalfNnz
// entries on: R-MAT 18 support (7.6M entries) by MSA 12.30 ms in full and 6.70
// by halves (of which the mirror takes 0.13), inner product 16.6 and 9.2 ms,
// hybrid 9.3 and 5.0; R-MAT 16 by MSA / MCA / merge 1.65 / 4.04 / 4.47 and
// 1.17 / 2.69 / 3.08 ms; at 426,000 entries MSA 457 and 384 us; at 110,000
// hybrid 407 and 437, inner product 122 and 144 us. A handle's first use pays
// for the check: 0.16 ms at R-MAT 18. A check holds for as long as nobody else
// can write the values: a matrix whose arrays' addresses the caller has asked
// for is multiplied in full, unless the caller declared it symmetric.
constexpr int64_t kSymHalfNnz = 1 << 18;

static bool mxm_symmetric(ga_ctx ctx, ga_csr A, ga_csr B, ga_csr M) {
    const bool one = A->rst == B->rst && A->col == B->col && A->val == B->val && A->rst == M->rst && A->col == M->col;
    if (!one || A->m != A->n || A->nnz < kSymHalfNnz) return false;
    if (A->lent && !A->declared) return false;
    if (A->sym >= 0) return A->sym == 1;
    // the check synchronises: not inside a stream capture
    cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
    if (cudaStreamIsCapturing(ctx->stream, &cap) != cudaSuccess || cap != cudaStreamCaptureStatusNone) {
        cudaGetLastError();
        return false;
    }
    return csr_is_symmetric(ctx, A);
}

void mxm_masked_into(ga_ctx ctx, ga_algo algo, ga_csr A, ga_csr B, ga_csr M, void* d_cvals) {
    GA_REQUIRE(A->n == B->m, GA_ERR_SHAPE, "mxm: A.n != B.m");
    GA_REQUIRE(M->m == A->m && M->n == B->n, GA_ERR_SHAPE, "mxm: mask shape differs from A*B");
    GA_REQUIRE(A->dtype == B->dtype, GA_ERR_DTYPE, "mxm: A and B dtypes differ");
    if (M->nnz == 0 || M->m == 0) return;
    TuneScope tscope(ctx);
    algo = resolve_mxm_algo(ctx, algo, A, B, M);
    if (algo == GA_TRI) {
        if (tri_applies(ctx, A, B, M)) {
            tri_masked_into(ctx, A, static_cast<int32_t*>(d_cvals));
            return;
        }
        algo = GA_HYBRID;
    }
    if (algo == GA_NAIVE) {
        naive_masked_into(ctx, A, B, M, d_cvals);
        return;
    }
    const bool unit_b = csr_unit_values(ctx, B);
    const bool unit_a = (unit_b || algo == GA_DOT) && csr_unit_values(ctx, A);
    const bool ones = unit_a && A->dtype == GA_INT32;
    if (mxm_symmetric(ctx, A, B, M)) {
        // the upper part of every row, then its mirror
        DBuf<int32_t> ust(ctx, (size_t)M->m + 1);
        upper_starts(ctx, A, ust.p);
        ga_csr_s Mu = *M;
        Mu.rst = ust.p;
        if (algo == GA_DOT) {
            mxm_dot_launch(ctx, A, B, B, &Mu, d_cvals, unit_a && unit_b, A->rst + 1, A->rst);
        } else {
            MxmRows rows;
            rows.counted = A->rst;
            DBuf<unsigned char> scratch(ctx, mxm_scratch_bytes(M->m, M->n, M->nnz, algo == GA_HYBRID));
            mxm_masked_launch(ctx, algo, A, B, &Mu, d_cvals, scratch.p, M->nnz, unit_b, A->rst + 1, ones,
                              algo == GA_HYBRID ? B : nullptr, rows);
        }
        mirror_values(ctx, A, d_cvals, A->dtype);
        return;
    }
    if (algo == GA_DOT || algo == GA_HYBRID) {
        const bool sym = csr_is_symmetric(ctx, B);
        ga_csr Bt = sym ? B : transpose_csr(ctx, B);
        try {
            if (algo == GA_DOT) {
                mxm_dot_launch(ctx, A, B, Bt, M, d_cvals, unit_a && unit_b, nullptr);
            } else {
                DBuf<unsigned char> scratch(ctx, mxm_scratch_bytes(M->m, M->n, M->nnz));
                mxm_masked_launch(ctx, GA_HYBRID, A, B, M, d_cvals, scratch.p, M->nnz, unit_b, nullptr, ones, Bt);
            }
        } catch (...) {
            if (!sym) csr_destroy(ctx, Bt);
            throw;
        }
        if (!sym) csr_destroy(ctx, Bt);
        return;
    }
    DBuf<unsigned char> scratch(ctx, mxm_scratch_bytes(M->m, M->n, M->nnz));
    mxm_masked_launch(ctx, algo, A, B, M, d_cvals, scratch.p, M->nnz, unit_b, nullptr, ones);
}

}  // namespace ga

using namespace ga;

extern "C" {

int ga_mxm_masked_vals(ga_ctx ctx, ga_algo algo, ga_csr A, ga_csr B, ga_csr M, void* d_cvals) {
    if (!ctx || !A || !B || !M || (!d_cvals && M->nnz)) return GA_ERR_INVALID_ARG;
    GA_API_BODY(ctx, mxm_masked_into(ctx, algo, A, B, M, d_cvals));
}

int ga_mxm_masked(ga_ctx ctx, ga_algo algo, ga_csr A, ga_csr B, ga_csr M, ga_csr* C) {
    if (!ctx || !A || !B || !M || !C) return GA_ERR_INVALID_ARG;
    *C = nullptr;
    GA_API_BODY(ctx, {
        GA_REQUIRE(A->dtype == B->dtype, GA_ERR_DTYPE, "mxm: A and B dtypes differ");
        ga_csr R = csr_alloc(ctx, M->m, M->n, M->nnz, A->dtype);
        try {
            GA_CUDA(cudaMemcpyAsync(R->rst, M->rst, sizeof(int32_t) * (M->m + 1), cudaMemcpyDeviceToDevice,
                                    ctx->stream));
            if (M->nnz)
                GA_CUDA(cudaMemcpyAsync(R->col, M->col, sizeof(int32_t) * M->nnz, cudaMemcpyDeviceToDevice,
                                        ctx->stream));
            mxm_masked_into(ctx, algo, A, B, M, R->val);
        } catch (...) {
            csr_destroy(ctx, R);
            throw;
        }
        *C = R;
    });
}

}  // extern "C"
