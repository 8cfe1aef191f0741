// sort.cu -- stable LSD radix sort and stable stream compaction.
//
// The reference orders each genDist output chunk with Thrust's device
// sort_by_key on float keys (genCUDA.cu:39-45), which is a stable radix sort,
// and orders kmerDist output by the host scan of whole tiles
// (kmerMain.cpp:175-195).  Both orders are reproduced here with one stable
// LSD radix sort written for this library:
//   * up to 8,192 items: one block sorts everything in registers and shared
//     memory, one launch;
//   * above: passes of at most 9 bits, as few as the key's bits allow and of
//     equal width, each a histogram per 4,096-item tile, an exclusive scan
//     (one warp per digit) and a stable scatter.
// Bound: launches and their gaps at a few thousand items, L2 traffic above.  With
// 4 to 7 passes of three launches whatever the size, sorts took 290 of the 708
// us of kernel time for 1,000 reads; a whole call went from 592 to 460 us, one of
// 200 alignments from 207 to 170, one of 20,000 reads from 2.09 to 1.94 ms.
// Ranks come from warp matches on the digit, counted per warp over the warp's
// own stretch of consecutive items.
#include <cuda_runtime.h>

#include <algorithm>

#include "internal.h"

namespace crispy {
namespace {

constexpr int kSortThreads = 256;
constexpr int kSortItems = 16;                       // per thread
constexpr int kSortTile = kSortThreads * kSortItems; // 4096
constexpr int kWarps = kSortThreads / 32;
constexpr int kMaxDigitBits = 9;
constexpr int kMaxBins = 1 << kMaxDigitBits;

// A warp's digit counts: lane's rank among the warp's items of the same digit
// so far.  All 32 lanes call it, in item order.
__device__ __forceinline__ uint32_t warp_rank(uint16_t* cnt, uint32_t d, int lane) {
    const uint32_t peers = __match_any_sync(0xffffffffu, d);
    const int leader = __ffs(peers) - 1;
    uint32_t at = 0;
    if (lane == leader) {
        at = cnt[d];
        cnt[d] = (uint16_t)(at + __popc(peers));
    }
    at = __shfl_sync(0xffffffffu, at, leader);
    __syncwarp();
    return at + __popc(peers & ((1u << lane) - 1u));
}

// Inclusive sum over the block (up to 1,024 threads) of one value a thread.
__device__ __forceinline__ uint32_t block_inclusive(uint32_t v, uint32_t* wsum, int nwarps) {
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = v;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    if (lane == 31) wsum[w] = x;
    __syncthreads();
    if (w == 0) {
        uint32_t z = lane < nwarps ? wsum[lane] : 0u;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, z, o);
            if (lane >= o) z += y;
        }
        wsum[lane] = z;
    }
    __syncthreads();
    return x + (w > 0 ? wsum[w - 1] : 0u);
}

// The whole sort in one block of 1,024 threads, kItems consecutive items a
// lane apart by 32, a warp's items consecutive.  Items past n carry the
// largest key and stay behind all others.
constexpr int kBlockThreads = 1024;
constexpr int kBlockBins = 256;
template <class K, bool kVals, int kItems>
__global__ void __launch_bounds__(kBlockThreads, 1) rs_block(const K* __restrict__ kin,
                                                             const uint32_t* __restrict__ vin,
                                                             K* __restrict__ kout, uint32_t* __restrict__ vout,
                                                             int n, int passes, int width) {
    extern __shared__ __align__(16) uint8_t smem[];
    __shared__ uint32_t wsum[32];
    constexpr int kN = kBlockThreads * kItems;
    K* sk = reinterpret_cast<K*>(smem);
    uint32_t* sv = reinterpret_cast<uint32_t*>(sk + kN);
    uint16_t* cnt = reinterpret_cast<uint16_t*>(sv + (kVals ? kN : 0));   // [32 warps][256]
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int first = w * 32 * kItems + lane;
    const uint32_t mask = (1u << width) - 1u;
    K key[kItems];
    uint32_t val[kItems];
#pragma unroll
    for (int j = 0; j < kItems; ++j) {
        const int i = first + 32 * j;
        key[j] = i < n ? kin[i] : ~K(0);
        val[j] = kVals && i < n ? vin[i] : 0u;
    }
    for (int p = 0; p < passes; ++p) {
        const int shift = p * width;
#pragma unroll
        for (int q = 0; q < 32 * kBlockBins / 8 / kBlockThreads; ++q)
            reinterpret_cast<uint4*>(cnt)[q * kBlockThreads + t] = make_uint4(0u, 0u, 0u, 0u);
        __syncthreads();
        uint32_t pos[kItems];
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            pos[j] = warp_rank(cnt + w * kBlockBins, (uint32_t)(key[j] >> shift) & mask, lane);
        __syncthreads();
        // exclusive sums in (digit, warp) order: thread t takes warps
        // 8 (t % 4) .. of digit t / 4
        uint32_t c[8], sum = 0;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            c[q] = cnt[(8 * (t & 3) + q) * kBlockBins + (t >> 2)];
            sum += c[q];
        }
        uint32_t run = block_inclusive(sum, wsum, 32) - sum;
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            cnt[(8 * (t & 3) + q) * kBlockBins + (t >> 2)] = (uint16_t)run;
            run += c[q];
        }
        __syncthreads();
#pragma unroll
        for (int j = 0; j < kItems; ++j)
            pos[j] += cnt[w * kBlockBins + ((uint32_t)(key[j] >> shift) & mask)];
        if (p + 1 < passes) {
#pragma unroll
            for (int j = 0; j < kItems; ++j) {
                sk[pos[j]] = key[j];
                if (kVals) sv[pos[j]] = val[j];
            }
            __syncthreads();
#pragma unroll
            for (int j = 0; j < kItems; ++j) {
                key[j] = sk[first + 32 * j];
                if (kVals) val[j] = sv[first + 32 * j];
            }
        } else {
#pragma unroll
            for (int j = 0; j < kItems; ++j) {
                if (pos[j] < (uint32_t)n) {
                    kout[pos[j]] = key[j];
                    if (kVals) vout[pos[j]] = val[j];
                }
            }
        }
    }
}

template <class K>
__global__ void __launch_bounds__(kSortThreads) rs_hist(const K* __restrict__ keys, int64_t n,
                                                        int shift, uint32_t mask, uint32_t* __restrict__ hist,
                                                        int nblocks) {
    __shared__ uint32_t cnt[kMaxBins];
    for (int d = threadIdx.x; d <= (int)mask; d += kSortThreads) cnt[d] = 0;
    __syncthreads();
    const int64_t base = (int64_t)blockIdx.x * kSortTile;
#pragma unroll 4
    for (int j = 0; j < kSortItems; ++j) {
        int64_t i = base + (int64_t)j * kSortThreads + threadIdx.x;
        if (i < n) atomicAdd(&cnt[(uint32_t)(keys[i] >> shift) & mask], 1u);
    }
    __syncthreads();
    for (int d = threadIdx.x; d <= (int)mask; d += kSortThreads) hist[(int64_t)d * nblocks + blockIdx.x] = cnt[d];
}

// One warp per digit: exclusive sums of its counts over the tiles, and their
// total.
__global__ void __launch_bounds__(256) rs_rows(uint32_t* __restrict__ hist, int nblocks, int bins,
                                               uint32_t* __restrict__ total) {
    const int lane = threadIdx.x & 31;
    const int d = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (d >= bins) return;
    uint32_t* row = hist + (int64_t)d * nblocks;
    uint32_t carry = 0;
    for (int b = 0; b < nblocks; b += 32) {
        const uint32_t v = b + lane < nblocks ? row[b + lane] : 0u;
        uint32_t x = v;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (b + lane < nblocks) row[b + lane] = carry + x - v;
        carry += __shfl_sync(0xffffffffu, x, 31);
    }
    if (lane == 0) total[d] = carry;
}

// Exclusive scan of m uint32 values in place with one block; writes the sum
// to *total when total != nullptr.  The block walks the array in tiles of
// 4096 values (four consecutive values per thread, coalesced), carrying the
// running sum from tile to tile.
__global__ void __launch_bounds__(1024) scan_exclusive_1blk(uint32_t* __restrict__ v, int64_t m,
                                                            uint32_t* __restrict__ total) {
    __shared__ uint32_t wsum[32];
    __shared__ uint32_t s_carry;
    const int t = threadIdx.x;
    const int lane = t & 31, w = t >> 5;
    if (t == 0) s_carry = 0;
    __syncthreads();
    const bool vec = (reinterpret_cast<uintptr_t>(v) & 15u) == 0;
    for (int64_t base = 0; base < m; base += 4096) {
        const int64_t i0 = base + 4 * (int64_t)t;
        uint32_t a[4];
        if (vec && i0 + 3 < m) {
            const uint4 q = *reinterpret_cast<const uint4*>(v + i0);
            a[0] = q.x; a[1] = q.y; a[2] = q.z; a[3] = q.w;
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) a[k] = i0 + k < m ? v[i0 + k] : 0u;
        }
        const uint32_t sum = a[0] + a[1] + a[2] + a[3];
        uint32_t x = sum;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
            if (lane >= o) x += y;
        }
        if (lane == 31) wsum[w] = x;
        __syncthreads();
        if (w == 0) {
            uint32_t z = wsum[lane];
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, z, o);
                if (lane >= o) z += y;
            }
            wsum[lane] = z;
        }
        __syncthreads();
        const uint32_t carry = s_carry;
        uint32_t run = carry + x - sum + (w > 0 ? wsum[w - 1] : 0u);
        uint32_t out[4];
#pragma unroll
        for (int k = 0; k < 4; ++k) { out[k] = run; run += a[k]; }
        if (vec && i0 + 3 < m) {
            *reinterpret_cast<uint4*>(v + i0) = make_uint4(out[0], out[1], out[2], out[3]);
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) if (i0 + k < m) v[i0 + k] = out[k];
        }
        __syncthreads();   // every thread has read s_carry and wsum
        if (t == 1023) s_carry = carry + wsum[31];
        __syncthreads();
    }
    if (t == 0 && total) *total = s_carry;
}

template <class K, bool kVals>
__global__ void __launch_bounds__(kSortThreads) rs_scatter(const K* __restrict__ kin,
                                                           const uint32_t* __restrict__ vin,
                                                           K* __restrict__ kout,
                                                           uint32_t* __restrict__ vout, int64_t n,
                                                           int shift, uint32_t mask,
                                                           const uint32_t* __restrict__ offs,
                                                           const uint32_t* __restrict__ total,
                                                           int nblocks) {
    __shared__ uint32_t base[kMaxBins];        // position of the tile's first item per digit
    __shared__ __align__(16) uint16_t cnt[kWarps][kMaxBins];
    __shared__ uint32_t wsum[32];
    const int t = threadIdx.x, lane = t & 31, w = t >> 5;
    const int bins = (int)mask + 1;
    const int64_t first = (int64_t)blockIdx.x * kSortTile + w * (32 * kSortItems) + lane;
    K key[kSortItems];
    uint32_t val[kSortItems], pos[kSortItems];
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        const int64_t i = first + 32 * j;
        key[j] = i < n ? kin[i] : ~K(0);       // past the end: behind all others of the last tile
        val[j] = kVals && i < n ? vin[i] : 0u;
    }
    for (int q = t; q < kWarps * kMaxBins / 8; q += kSortThreads)
        reinterpret_cast<uint4*>(cnt)[q] = make_uint4(0u, 0u, 0u, 0u);
    {
        // digits' first positions: exclusive sums of the totals, two a thread
        const uint32_t a0 = 2 * t < bins ? total[2 * t] : 0u, a1 = 2 * t + 1 < bins ? total[2 * t + 1] : 0u;
        const uint32_t x = block_inclusive(a0 + a1, wsum, kWarps) - a0 - a1;
        if (2 * t < bins) base[2 * t] = x + offs[(int64_t)(2 * t) * nblocks + blockIdx.x];
        if (2 * t + 1 < bins) base[2 * t + 1] = x + a0 + offs[(int64_t)(2 * t + 1) * nblocks + blockIdx.x];
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) pos[j] = warp_rank(cnt[w], (uint32_t)(key[j] >> shift) & mask, lane);
    __syncthreads();
    for (int d = t; d < bins; d += kSortThreads) {
        uint32_t run = 0;
#pragma unroll
        for (int q = 0; q < kWarps; ++q) {
            const uint32_t c = cnt[q][d];
            cnt[q][d] = (uint16_t)run;
            run += c;
        }
    }
    __syncthreads();
#pragma unroll
    for (int j = 0; j < kSortItems; ++j) {
        if (first + 32 * j < n) {
            const uint32_t d = (uint32_t)(key[j] >> shift) & mask;
            const uint32_t at = base[d] + cnt[w][d] + pos[j];
            kout[at] = key[j];
            if (kVals) vout[at] = val[j];
        }
    }
}

// Passes and bits per pass of a sort.
struct SortPlan {
    bool block;
    int passes, width;
};
constexpr int kBlockMax = 8192;   // beyond: one block per 4,096 items beats one block for all
SortPlan sort_plan(int64_t n, int key_bits) {
    SortPlan p;
    p.block = n <= kBlockMax;
    const int most = p.block ? 8 : kMaxDigitBits;
    const int bits = std::max(1, key_bits);
    p.passes = (bits + most - 1) / most;
    p.width = (bits + p.passes - 1) / p.passes;
    return p;
}

template <class K, bool kVals, int kItems>
int block_sort(crispy_ctx* ctx, cudaStream_t s, const K* keys, const uint32_t* vals, K* kout, uint32_t* vout,
               int n, const SortPlan& p) {
    const size_t smem = (size_t)kBlockThreads * kItems * (sizeof(K) + (kVals ? 4 : 0)) + 32 * kBlockBins * 2;
    auto fn = rs_block<K, kVals, kItems>;
    CRISPY_CK(ctx, cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    fn<<<1, kBlockThreads, smem, s>>>(keys, vals, kout, vout, n, p.passes, p.width);
    count_launch(ctx);
    CRISPY_CK(ctx, cudaGetLastError());
    return CRISPY_OK;
}

template <class K, bool kVals>
int radix_sort(crispy_ctx* ctx, cudaStream_t s, K* keys, K* keys_alt, uint32_t* vals,
               uint32_t* vals_alt, int64_t n, int key_bits, K** out_keys, uint32_t** out_vals,
               DevBuf& tmp) {
    const bool alt = sort_lands_in_alt(n, key_bits);
    *out_keys = alt ? keys_alt : keys;
    if (out_vals) *out_vals = alt ? vals_alt : vals;
    if (n <= 1) return CRISPY_OK;
    const SortPlan p = sort_plan(n, key_bits);
    if (p.block) {
        if (n <= 2 * kBlockThreads)
            return block_sort<K, kVals, 2>(ctx, s, keys, vals, keys_alt, vals_alt, (int)n, p);
        return block_sort<K, kVals, kBlockMax / kBlockThreads>(ctx, s, keys, vals, keys_alt, vals_alt, (int)n, p);
    }
    const int nblocks = (int)((n + kSortTile - 1) / kSortTile);
    const int bins = 1 << p.width;
    CRISPY_TRY(ensure(ctx, tmp, sort_tmp_bytes(n)));
    uint32_t* total = tmp.as<uint32_t>();
    uint32_t* hist = total + kMaxBins;
    K *src = keys, *dst = keys_alt;
    uint32_t *vsrc = vals, *vdst = vals_alt;
    for (int q = 0; q < p.passes; ++q) {
        const int shift = q * p.width;
        rs_hist<K><<<nblocks, kSortThreads, 0, s>>>(src, n, shift, (uint32_t)bins - 1u, hist, nblocks);
        rs_rows<<<(bins + 7) / 8, 256, 0, s>>>(hist, nblocks, bins, total);
        rs_scatter<K, kVals><<<nblocks, kSortThreads, 0, s>>>(src, vsrc, dst, vdst, n, shift, (uint32_t)bins - 1u,
                                                              hist, total, nblocks);
        count_launch(ctx, 3);
        std::swap(src, dst);
        std::swap(vsrc, vdst);
    }
    CRISPY_CK(ctx, cudaGetLastError());
    return CRISPY_OK;
}

constexpr int kCmpThreads = 256;
constexpr int kCmpPer = kScanTile / kCmpThreads;  // 18
static_assert(kScanTile % kCmpThreads == 0, "tile");

__global__ void __launch_bounds__(kCmpThreads) cmp_count(const uint8_t* __restrict__ flags,
                                                         int64_t n, uint32_t* __restrict__ cnt) {
    const int64_t base = (int64_t)blockIdx.x * kScanTile;
    uint32_t c = 0;
    for (int j = 0; j < kCmpPer; ++j) {
        int64_t i = base + (int64_t)j * kCmpThreads + threadIdx.x;
        if (i < n) c += flags[i] != 0;
    }
    c = __reduce_add_sync(0xffffffffu, c);
    __shared__ uint32_t ws[kCmpThreads / 32];
    if ((threadIdx.x & 31) == 0) ws[threadIdx.x >> 5] = c;
    __syncthreads();
    if (threadIdx.x == 0) {
        uint32_t s = 0;
        for (int q = 0; q < kCmpThreads / 32; ++q) s += ws[q];
        cnt[blockIdx.x] = s;
    }
}

// Each thread owns kCmpPer consecutive items, so output order is item order.
__global__ void __launch_bounds__(kCmpThreads) cmp_scatter(const uint8_t* __restrict__ flags,
                                                           int64_t n,
                                                           const uint32_t* __restrict__ offs,
                                                           uint32_t* __restrict__ out) {
    const int64_t base = (int64_t)blockIdx.x * kScanTile + (int64_t)threadIdx.x * kCmpPer;
    uint32_t mine = 0;
    uint32_t bits = 0;
#pragma unroll
    for (int j = 0; j < kCmpPer; ++j) {
        int64_t i = base + j;
        uint32_t f = (i < n) ? (flags[i] != 0) : 0u;
        bits |= f << j;
        mine += f;
    }
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    uint32_t x = mine;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    __shared__ uint32_t ws[kCmpThreads / 32];
    if (lane == 31) ws[w] = x;
    __syncthreads();
    uint32_t wbase = 0;
    for (int q = 0; q < w; ++q) wbase += ws[q];
    uint32_t pos = offs[blockIdx.x] + wbase + x - mine;
    while (bits) {
        int j = __ffs(bits) - 1;
        bits &= bits - 1;
        out[pos++] = (uint32_t)(base + j);
    }
}

}  // namespace

size_t sort_tmp_bytes(int64_t n) {
    const int64_t nblocks = (n + kSortTile - 1) / kSortTile;
    return (size_t)kMaxBins * (size_t)(std::max<int64_t>(nblocks, 1) + 1) * sizeof(uint32_t);
}

bool sort_lands_in_alt(int64_t n, int key_bits) {
    if (n <= 1) return false;
    const SortPlan p = sort_plan(n, key_bits);
    return p.block || (p.passes & 1);
}

int sort_u64_payload(crispy_ctx* ctx, cudaStream_t s, uint64_t* keys, uint64_t* keys_alt,
                     uint32_t* vals, uint32_t* vals_alt, int64_t n, int key_bits, bool with_vals,
                     uint64_t** sorted_keys, uint32_t** sorted_vals, DevBuf& tmp) {
    if (with_vals)
        return radix_sort<uint64_t, true>(ctx, s, keys, keys_alt, vals, vals_alt, n, key_bits,
                                          sorted_keys, sorted_vals, tmp);
    return radix_sort<uint64_t, false>(ctx, s, keys, keys_alt, nullptr, nullptr, n, key_bits,
                                       sorted_keys, nullptr, tmp);
}

int sort_u32_payload(crispy_ctx* ctx, cudaStream_t s, uint32_t* keys, uint32_t* keys_alt,
                     uint32_t* vals, uint32_t* vals_alt, int64_t n, int key_bits,
                     uint32_t** sorted_keys, uint32_t** sorted_vals, DevBuf& tmp) {
    return radix_sort<uint32_t, true>(ctx, s, keys, keys_alt, vals, vals_alt, n, key_bits,
                                      sorted_keys, sorted_vals, tmp);
}

int compact_flags(crispy_ctx* ctx, cudaStream_t s, const uint8_t* flags, int64_t n,
                  uint32_t* out_idx, uint32_t* tile_counts, DevBuf& tmp, int64_t* total) {
    if (total) *total = 0;
    if (n <= 0) return CRISPY_OK;
    const int nt = (int)((n + kScanTile - 1) / kScanTile);
    CRISPY_TRY(ensure(ctx, tmp, (size_t)(nt + 1) * sizeof(uint32_t)));
    uint32_t* offs = tmp.as<uint32_t>();
    cmp_count<<<nt, kCmpThreads, 0, s>>>(flags, n, tile_counts);
    CRISPY_CK(ctx, cudaMemcpyAsync(offs, tile_counts, nt * sizeof(uint32_t),
                                   cudaMemcpyDeviceToDevice, s));
    scan_exclusive_1blk<<<1, 1024, 0, s>>>(offs, nt, offs + nt);
    cmp_scatter<<<nt, kCmpThreads, 0, s>>>(flags, n, offs, out_idx);
    count_launch(ctx, 3);
    CRISPY_CK(ctx, cudaGetLastError());
    if (!total) return CRISPY_OK;   // the caller reads tile_counts (and sums them) itself
    uint32_t tot = 0;
    CRISPY_CK(ctx, cudaMemcpyAsync(&tot, offs + nt, sizeof(uint32_t), cudaMemcpyDeviceToHost, s));
    CRISPY_CK(ctx, cudaStreamSynchronize(s));
    *total = tot;
    return CRISPY_OK;
}

}  // namespace crispy
