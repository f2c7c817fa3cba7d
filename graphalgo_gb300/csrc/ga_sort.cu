// Stable least-significant-digit radix sort of integer keys with an optional
// int32 payload: the order behind edge lists to CSR (keys row and column) and
// the transpose (keys the columns of a CSR).
//
// Per pass over one digit (up to kDigitBits bits): the tiles' digit counts,
// their scan over (digit, tile), then every tile ranks its keys and writes
// them. A tile's keys are ranked in order (warps take consecutive stretches,
// 32 keys at a time; lanes with equal digits are found by one ballot per digit
// bit), gathered by digit in shared memory and written from there, so that
// equal digits leave as one contiguous run. Bound by HBM and the L2: each pass
// reads the keys twice and writes them once. Few wide digits beat many narrow
// ones as long as the runs stay long: 8.4M 36-bit keys in 4 passes of 9 bits.
#include "ga_device.cuh"

#include <algorithm>

namespace ga {

constexpr int kRadixThreads = 256;
constexpr int kRadixWarps = kRadixThreads / 32;
constexpr int kRadixPer = 16;  // keys per thread
constexpr int kRadixTile = kRadixThreads * kRadixPer;
constexpr int kDigitBits = 10;

template <typename K>
__global__ void __launch_bounds__(kRadixThreads) k_radix_count(const K* __restrict__ keys, int64_t n, int shift,
                                                               int bits, int64_t tiles, int32_t* __restrict__ counts) {
    __shared__ int32_t h[1 << kDigitBits];
    const int bins = 1 << bits;
    for (int d = threadIdx.x; d < bins; d += kRadixThreads) h[d] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kRadixTile;
#pragma unroll
    for (int r = 0; r < kRadixPer; ++r) {
        const int64_t i = base + r * kRadixThreads + threadIdx.x;
        if (i < n) atomicAdd(&h[(int)(keys[i] >> shift) & (bins - 1)], 1);
    }
    __syncthreads();
    for (int d = threadIdx.x; d < bins; d += kRadixThreads) counts[d * tiles + blockIdx.x] = h[d];
}

// Shared memory: per warp and digit a counter, then the digits' first places
// in the tile, their places in the output, and the keys and payloads by digit.
template <typename K>
static size_t radix_smem(int bits, bool pay) {
    return (size_t)(1 << bits) * (kRadixWarps + 2) * sizeof(int32_t) +
           (size_t)kRadixTile * (sizeof(K) + (pay ? sizeof(int32_t) : 0));
}

template <typename K, bool PAY>
__global__ void __launch_bounds__(kRadixThreads) k_radix_scatter(const K* __restrict__ keys,
                                                                 const int32_t* __restrict__ pay, int64_t n, int shift,
                                                                 int bits, int64_t tiles,
                                                                 const int32_t* __restrict__ place,
                                                                 K* __restrict__ out, int32_t* __restrict__ out_pay) {
    extern __shared__ __align__(16) unsigned char smem[];
    const unsigned FULL = 0xffffffffu;
    const int bins = 1 << bits;
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    K* s_key = reinterpret_cast<K*>(smem);
    int32_t* s_pay = reinterpret_cast<int32_t*>(s_key + kRadixTile);
    int32_t* s_cnt = s_pay + (PAY ? kRadixTile : 0);  // [warp][digit]
    int32_t* s_first = s_cnt + kRadixWarps * bins;
    int32_t* s_place = s_first + bins;
    __shared__ int s_tot[kRadixWarps];
    for (int d = threadIdx.x; d < kRadixWarps * bins; d += kRadixThreads) s_cnt[d] = 0;
    for (int d = threadIdx.x; d < bins; d += kRadixThreads) s_place[d] = place[d * tiles + blockIdx.x];
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kRadixTile;
    const int count = (int)min((int64_t)kRadixTile, n - base);
    int32_t* my = s_cnt + wid * bins;
    K key[kRadixPer];
    int32_t rank[kRadixPer];
#pragma unroll
    for (int r = 0; r < kRadixPer; ++r) {
        const int i = wid * (kRadixPer * 32) + r * 32 + lane;
        key[r] = i < count ? keys[base + i] : (K)0;
    }
#pragma unroll
    for (int r = 0; r < kRadixPer; ++r) {
        const int i = wid * (kRadixPer * 32) + r * 32 + lane;
        const int d = (int)(key[r] >> shift) & (bins - 1);
        unsigned same = __ballot_sync(FULL, i < count);  // lanes with this lane's digit
        for (int b = 0; b < bits; ++b) {
            const bool one = d >> b & 1;
            const unsigned v = __ballot_sync(FULL, one);
            same &= one ? v : ~v;
        }
        if (i < count) rank[r] = my[d] + __popc(same & ((1u << lane) - 1u));
        __syncwarp();
        if (i < count && (same & ((1u << lane) - 1u)) == 0u) my[d] += __popc(same);
        __syncwarp();
    }
    __syncthreads();
    // per digit: the warps' counts to first places, and the digits' totals
    // scanned over the tile; thread t owns the digits t * per ...
    const int per = (bins + kRadixThreads - 1) / kRadixThreads;
    int mine = 0;
    for (int x = 0; x < per; ++x) {
        const int d = threadIdx.x * per + x;
        if (d >= bins) break;
        int run = 0;
        for (int w = 0; w < kRadixWarps; ++w) {
            const int c = s_cnt[w * bins + d];
            s_cnt[w * bins + d] = run;
            run += c;
        }
        s_first[d] = mine;
        mine += run;
    }
    const int incl = warp_incl_scan(mine);
    if (lane == 31) s_tot[wid] = incl;
    __syncthreads();
    int before = incl - mine;
    for (int w = 0; w < wid; ++w) before += s_tot[w];
    for (int x = 0; x < per; ++x) {
        const int d = threadIdx.x * per + x;
        if (d < bins) s_first[d] += before;
    }
    __syncthreads();
#pragma unroll
    for (int r = 0; r < kRadixPer; ++r) {
        const int i = wid * (kRadixPer * 32) + r * 32 + lane;
        if (i < count) {
            const int d = (int)(key[r] >> shift) & (bins - 1);
            const int at = s_first[d] + my[d] + rank[r];
            s_key[at] = key[r];
            if (PAY) s_pay[at] = pay[base + i];
        }
    }
    __syncthreads();
    for (int i = threadIdx.x; i < count; i += kRadixThreads) {
        const K k = s_key[i];
        const int d = (int)(k >> shift) & (bins - 1);
        const int64_t to = (int64_t)s_place[d] + (i - s_first[d]);
        out[to] = k;
        if (PAY) out_pay[to] = s_pay[i];
    }
}

int64_t radix_sort_bytes(int64_t n) {
    const int64_t cells = ((n + kRadixTile - 1) / kRadixTile) << kDigitBits;
    return sizeof(int32_t) * (cells + 1) + (int64_t)scan_scratch_bytes(cells);
}

template <typename K>
static bool radix_sort(ga_ctx ctx, K* keys, K* tkeys, int32_t* pay, int32_t* tpay, int64_t n, int bits) {
    if (n <= 1 || bits <= 0) return false;
    ProfScope ps(ctx, "radix_sort");
    const int passes = (bits + kDigitBits - 1) / kDigitBits;
    const int64_t tiles = (n + kRadixTile - 1) / kRadixTile;
    const int width = (bits + passes - 1) / passes;
    const int64_t cells = tiles << width;
    DBuf<int32_t> counts(ctx, (size_t)cells + 1);
    DBuf<char> scr(ctx, scan_scratch_bytes(cells));
    auto scatter = pay ? k_radix_scatter<K, true> : k_radix_scatter<K, false>;
    const size_t smem = radix_smem<K>(width, pay != nullptr);
    // the attribute is the kernel's, shared by concurrent calls: always the
    // size of the widest digit
    GA_CUDA(cudaFuncSetAttribute(scatter, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)radix_smem<K>(kDigitBits, pay != nullptr)));
    for (int p = 0; p < passes; ++p) {
        const int shift = p * width, b = std::min(width, bits - shift);
        k_radix_count<K><<<(unsigned)tiles, kRadixThreads, 0, ctx->stream>>>(keys, n, shift, b, tiles, counts.p);
        post_launch("radix_count");
        scan_exclusive_i32_scratch(ctx, counts.p, counts.p, tiles << b, scr.p);
        scatter<<<(unsigned)tiles, kRadixThreads, smem, ctx->stream>>>(keys, pay, n, shift, b, tiles, counts.p, tkeys,
                                                                      tpay);
        post_launch("radix_scatter");
        std::swap(keys, tkeys);
        std::swap(pay, tpay);
    }
    return passes & 1;
}

bool radix_sort_u64(ga_ctx ctx, uint64_t* keys, uint64_t* tkeys, int32_t* pay, int32_t* tpay, int64_t n, int bits) {
    return radix_sort<uint64_t>(ctx, keys, tkeys, pay, tpay, n, bits);
}

bool radix_sort_u32(ga_ctx ctx, uint32_t* keys, uint32_t* tkeys, int32_t* pay, int32_t* tpay, int64_t n, int bits) {
    return radix_sort<uint32_t>(ctx, keys, tkeys, pay, tpay, n, bits);
}

}  // namespace ga
