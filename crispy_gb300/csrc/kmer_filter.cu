// kmer_filter.cu -- kmerDist's candidate pairs on the tensor cores.
//
// The cut keeps a pair only if its reads share almost all their K-mers, and
// almost no pair does (1.2e-4 of the pairs of 99,999 reads of 300-500 nt).
// So the batched form at K >= 5 first bounds every pair from above with one
// contraction on the tensor cores, and counts exactly only the few pairs the
// bound leaves:
//   * every read's K-mer counts are folded into D bins (filter_map_kernel:
//     the K-mers of a sample in order of frequency, dealt to the bins back
//     and forth, so that all bins are about equally full).  With f the folded
//     counts, m(a, b) = sum_k min(c_a[k], c_b[k]) <= sum_d min(f_a[d], f_b[d]);
//   * min(x, y) <= sqrt(x y), so with g(f) the smallest e2m1 value >= sqrt(f)
//     (0, 1, 1.5, 2, 3, 4, 6) the signature g(f_a) gives
//         m(a, b) <= S(a, b) = sum_d g(f_a[d]) g(f_b[d]),
//     a dot product of 4-bit floats.  Counts beyond 36 = 6 * 6 are made up
//     for by the read's excess x = sum_d max(0, f[d] - 36): m <= S + x_a;
//   * every product is a multiple of 1/4 and every sum of a read of at most
//     2,048 nt stays below 2^18, so S is exact in the FP32 accumulator (the
//     compare leaves half a count of slack all the same);
//   * a pair whose S falls short of the cut's smallest count is dropped; the
//     others ("candidates") get their exact count from filter_verify_kernel,
//     and the cut's own integer test decides.  The survivors are the same
//     bits, whatever D and the fold.
// At K = 8 the reads are in the order of their H keys (kmer.cu) and the row
// panels cover only the columns that share a key with one of their rows,
// unless a read is H-heavy.
#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>
#include <vector>

#include "internal.h"
#include "kmer_emit.h"

namespace crispy {
namespace {

// ---- small device helpers -------------------------------------------------

// K-mer at position p of a 2-bit packed read (16 symbols per word, first
// symbol in the top bits; one word beyond the read must be readable).
__device__ __forceinline__ uint32_t packed_kmer(const uint32_t* w, int p, int K) {
    const int i = p >> 4;
    return __funnelshift_l(w[i + 1], w[i], 2 * (p & 15)) >> (32 - 2 * K);
}

// Two-bit codes (A0 G1 T2 C3, others 0) of four ASCII bases, first base in
// bits 7..6.
__device__ __forceinline__ uint32_t pack4(uint32_t x) {
    const uint32_t g = __vcmpeq4(x, 0x47474747u) & 0x01010101u;
    const uint32_t t = __vcmpeq4(x, 0x54545454u) & 0x02020202u;
    const uint32_t c = __vcmpeq4(x, 0x43434343u) & 0x03030303u;
    return ((g | t | c) * 0x40100401u) >> 24;
}

constexpr int kPackWarps = 8;

// One warp per read: ASCII to 2-bit words (the reads' bytes through aligned
// 32-bit loads and a funnel shift, four bases per load).  At K = 8 also the
// read order's sort key: (largest K-mer >= 0x8000, its count) << tbits | T.
__global__ void __launch_bounds__(kPackWarps * 32) filter_pack_kernel(
    const uint8_t* __restrict__ seq, const int64_t* __restrict__ off, const int32_t* __restrict__ tcount,
    int n, int K, int stride, uint32_t* packed, int tbits, uint64_t* __restrict__ keys,
    uint32_t* __restrict__ idx) {
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int nw = gridDim.x * kPackWarps;
    for (int r = blockIdx.x * kPackWarps + (threadIdx.x >> 5); r < n; r += nw) {
        const int T = tcount[r];
        const int L = T + K - 1;
        const uint8_t* s = seq + off[r];
        const uint32_t lead = (uint32_t)(reinterpret_cast<uintptr_t>(s) & 3u);
        const uint32_t* base = reinterpret_cast<const uint32_t*>(s - lead);
        uint32_t* dst = packed + (int64_t)r * stride;
        for (int w = lane; w < stride; w += 32) {
            const int p0 = 16 * w;
            uint32_t word = 0;
            if (p0 < L) {
                uint32_t x[5];
#pragma unroll
                for (int i = 0; i < 5; ++i) x[i] = p0 + 4 * i < L + (int)lead ? __ldg(base + p0 / 4 + i) : 0u;
#pragma unroll
                for (int i = 0; i < 4; ++i)
                    word |= pack4(__funnelshift_r(x[i], x[i + 1], 8 * lead)) << (24 - 8 * i);
                if (L - p0 < 16) word &= ~0u << (32 - 2 * (L - p0));
            }
            dst[w] = word;
        }
        if (keys != nullptr) {
            __syncwarp();
            uint32_t hm = 0;
            for (int p = lane; p < T; p += 32) {
                const uint32_t v = packed_kmer(dst, p, 8);
                if (v >= 0x8000u) hm = max(hm, v);
            }
            hm = __reduce_max_sync(full, hm);
            uint32_t c = 0;
            if (hm != 0u)
                for (int p = lane; p < T; p += 32) c += packed_kmer(dst, p, 8) == hm;
            c = __reduce_add_sync(full, c);
            if (lane == 0) {
                const uint32_t key = hm != 0u ? (hm << 16) | (c & 0xFFFFu) : 0u;
                keys[r] = ((uint64_t)key << tbits) | (uint32_t)T;
                idx[r] = (uint32_t)r;
            }
        }
    }
}

// K = 8: per position of the read order its read ID, tuple count and H key.
__global__ void filter_order_kernel(const uint64_t* __restrict__ keys, const uint32_t* __restrict__ idx, int n,
                                    int tbits, int32_t* __restrict__ perm, int32_t* __restrict__ tpos,
                                    uint32_t* __restrict__ hkey) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const uint64_t k = keys[i];
    perm[i] = (int32_t)idx[i];
    tpos[i] = (int32_t)(k & ((1ull << tbits) - 1));
    hkey[i] = (uint32_t)(k >> tbits);
}

// K-mer frequencies of a sample of reads (every read of a small set).
__global__ void __launch_bounds__(256) filter_hist_kernel(const uint32_t* __restrict__ packed, int stride,
                                                          const int32_t* __restrict__ tcount, int n, int K,
                                                          int sample, uint32_t* __restrict__ hist) {
    const int lane = threadIdx.x & 31;
    const int i = blockIdx.x * 8 + (threadIdx.x >> 5);
    if (i >= sample) return;
    const int r = (int)((int64_t)i * n / sample);
    const uint32_t* w = packed + (int64_t)r * stride;
    for (int p = lane; p < tcount[r]; p += 32) atomicAdd(&hist[packed_kmer(w, p, K)], 1u);
}

// The fold: K-mers in descending order of (log-quantised) frequency, dealt
// to the D bins back and forth.  One block.
constexpr int kFreqBuckets = 264;
__device__ __forceinline__ int freq_bucket(uint32_t f) {
    if (f == 0) return 0;
    const int e = 31 - __clz(f);
    return 1 + 8 * e + (int)((f << (31 - e)) >> 28 & 7u);
}
__global__ void __launch_bounds__(1024) filter_map_kernel(const uint32_t* __restrict__ hist, int K4, int D,
                                                          uint16_t* __restrict__ map) {
    __shared__ uint32_t cnt[kFreqBuckets];
    const int lane = threadIdx.x & 31;
    for (int i = threadIdx.x; i < kFreqBuckets; i += 1024) cnt[i] = 0;
    __syncthreads();
    for (int k = threadIdx.x; k < K4; k += 1024) {
        const int b = freq_bucket(hist[k]);
        const unsigned act = __activemask();
        const unsigned peers = __match_any_sync(act, b);
        if (lane == __ffs(peers) - 1) atomicAdd(&cnt[b], (uint32_t)__popc(peers));
    }
    __syncthreads();
    if (threadIdx.x < 32) {   // exclusive sums from the most frequent bucket down
        uint32_t carry = 0;
        for (int c = 0; c < (kFreqBuckets + 31) / 32; ++c) {
            const int b = kFreqBuckets - 1 - (32 * c + lane);
            const uint32_t v = b >= 0 ? cnt[b] : 0u;
            uint32_t x = v;
#pragma unroll
            for (int o = 1; o < 32; o <<= 1) {
                const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
                if (lane >= o) x += y;
            }
            if (b >= 0) cnt[b] = carry + x - v;
            carry += __shfl_sync(0xffffffffu, x, 31);
        }
    }
    __syncthreads();
    for (int k = threadIdx.x; k < K4; k += 1024) {
        const int b = freq_bucket(hist[k]);
        const unsigned act = __activemask();
        const unsigned peers = __match_any_sync(act, b);
        const int leader = __ffs(peers) - 1;
        uint32_t rank = 0;
        if (lane == leader) rank = atomicAdd(&cnt[b], (uint32_t)__popc(peers));
        rank = __shfl_sync(peers, rank, leader) + __popc(peers & ((1u << lane) - 1u));
        const uint32_t row = rank / (uint32_t)D, col = rank - row * (uint32_t)D;
        map[k] = (uint16_t)((row & 1u) ? (uint32_t)D - 1u - col : col);
    }
}

// e2m1 code of the smallest 4-bit float >= sqrt(f) (f <= 36; 6 beyond).
__device__ __forceinline__ uint32_t sig_code(uint32_t f) {
    // f: 0 1 2 3 4 5..9 10..15 -> 0 1 1.5 2 2 3 4
    if (f < 16u) return (uint32_t)(0x6666665555544320ull >> (4u * f)) & 15u;
    return f == 16u ? 6u : 7u;
}

constexpr int kSigWarps = 8;

// One warp per position: its read's folded counts (two 16-bit counters per
// shared word), then the signature, 8 dimensions per 32-bit store.
__global__ void __launch_bounds__(kSigWarps * 32) filter_sig_kernel(
    const uint32_t* __restrict__ packed, int stride, const int32_t* __restrict__ tcount,
    const int32_t* __restrict__ perm, int n, int K, int D, const uint16_t* __restrict__ map,
    uint32_t* __restrict__ sig, uint16_t* __restrict__ excess, uint16_t* __restrict__ nh) {
    extern __shared__ __align__(16) uint32_t fold_words[];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    uint32_t* cnt = fold_words + (threadIdx.x >> 5) * (D / 2);
    for (int i = lane; i < D / 2; i += 32) cnt[i] = 0;
    __syncwarp();
    const int nw = gridDim.x * kSigWarps;
    for (int i = blockIdx.x * kSigWarps + (threadIdx.x >> 5); i < n; i += nw) {
        const int T = tcount[i];
        const uint32_t* w = packed + (int64_t)(perm ? perm[i] : i) * stride;
        uint32_t high = 0;
        for (int p = lane; p < T; p += 32) {
            const uint32_t v = packed_kmer(w, p, K);
            high += v >= 0x8000u;
            const uint32_t d = __ldg(map + v);
            atomicAdd(&cnt[d >> 1], 1u << (16u * (d & 1u)));
        }
        __syncwarp();
        uint32_t x = 0;
        for (int g = lane; g < D / 8; g += 32) {
            uint32_t word = 0;
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const uint32_t c = cnt[4 * g + q];
                cnt[4 * g + q] = 0;
                const uint32_t lo = c & 0xFFFFu, hi = c >> 16;
                word |= (sig_code(lo) | sig_code(hi) << 4) << (8 * q);
                x += (lo > 36u ? lo - 36u : 0u) + (hi > 36u ? hi - 36u : 0u);
            }
            sig[(int64_t)i * (D / 8) + g] = word;
        }
        x = __reduce_add_sync(full, x);
        if (nh != nullptr) high = __reduce_add_sync(full, high);
        if (lane == 0) {
            excess[i] = (uint16_t)min(x, 0xFFFFu);
            if (nh != nullptr) nh[i] = (uint16_t)high;
        }
        __syncwarp();
    }
}

// Control block of a pass (device): candidate counts per round, then flags.
constexpr int kMaxRounds = 72;
struct FilterCtl {
    unsigned long long cand[kMaxRounds];
    uint32_t cursor[kMaxRounds];   // sorted candidates handed out, per round
    uint32_t overflow;    // the candidates are too many
    uint32_t timeout;     // a bounded wait ran out
    uint32_t any_heavy;   // K = 8: a read is H-heavy
    uint32_t pad;
};

// True once a round's candidates outgrew the buffer (or will) or a wait ran
// out: the kernels that follow have nothing to do.
__device__ __forceinline__ bool pass_ended(const FilterCtl* ctl) {
    return (*reinterpret_cast<const volatile uint32_t*>(&ctl->overflow) |
            *reinterpret_cast<const volatile uint32_t*>(&ctl->timeout)) != 0;
}

// After the probe: its candidates against what its share of the tiles may have.
__device__ __forceinline__ bool probe_says_too_many(FilterCtl* ctl, unsigned long long most) {
    const bool too_many = ctl->cand[0] > most;
    if (too_many && blockIdx.x == 0 && threadIdx.x == 0) ctl->overflow = 1u;
    return too_many;
}
__global__ void filter_probe_kernel(FilterCtl* ctl, unsigned long long most) { probe_says_too_many(ctl, most); }

// ---- exact lists --------------------------------------------------------------
// For the exact count every read is two lists: its distinct K-mers (16 bits
// each, padded to a multiple of 8 with copies of the first) and its repeats,
// one word (rank << 16 | K-mer) for each further occurrence (rank >= 1).  With
// both reads' lists, m = #(distinct K-mers of b in a) + #(repeats of b in a).
constexpr int kListWarps = 8;
constexpr uint32_t kSlotEmpty = 0xFFFFFFFFu;

// One warp per position.  Occurrence ranks come from a counter table in
// shared memory: direct (two 16-bit counters per word) up to K = 6, an
// open-addressing table (K-mer << 16 | count, load at most 1/2) above.
// The lists come between the probe and the rest of the pass and look at its
// candidates, of which there may be `most`.
// Repeats take the next free words of one array, whose size bounds them all;
// up to kStaged of a read's are collected on the way (a second pass over the
// read's distinct K-mers for them cost as much as the first).
constexpr int kStaged = 96;
template <bool kDirect>
__global__ void __launch_bounds__(kListWarps * 32) filter_lists_kernel(
    const uint32_t* __restrict__ packed, int stride, const int32_t* __restrict__ tcount,
    const int32_t* __restrict__ perm, int n, int K, int words, int hshift, uint16_t* __restrict__ distinct,
    int dstride, int4* __restrict__ meta, uint32_t* __restrict__ repeats, uint32_t* cursor, FilterCtl* ctl,
    unsigned long long most) {
    if (probe_says_too_many(ctl, most) || pass_ended(ctl)) return;
    extern __shared__ __align__(16) uint32_t tables[];
    __shared__ uint32_t staged_all[kListWarps][kStaged];
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const uint32_t lt = (1u << lane) - 1u;
    uint32_t* staged = staged_all[threadIdx.x >> 5];
    uint32_t* tbl = tables + (threadIdx.x >> 5) * words;
    const uint32_t blank = kDirect ? 0u : kSlotEmpty;
    const int nw = gridDim.x * kListWarps;
    for (int i = blockIdx.x * kListWarps + (threadIdx.x >> 5); i < n; i += nw) {
        const int T = tcount[i];
        const uint32_t* w = packed + (int64_t)(perm ? perm[i] : i) * stride;
        uint16_t* dst = distinct + (int64_t)i * dstride;
        for (int q = lane; q < words / 4; q += 32)
            reinterpret_cast<uint4*>(tbl)[q] = make_uint4(blank, blank, blank, blank);
        __syncwarp();
        int nd = 0, nr = 0;
        uint32_t first = 0;
        for (int p0 = 0; p0 < T; p0 += 32) {
            const int p = p0 + lane;
            uint32_t v = 0, rank = 0xFFFFu;
            if (p < T) {
                v = packed_kmer(w, p, K);
                if (kDirect) {
                    const uint32_t sh = 16u * (v & 1u);
                    rank = (atomicAdd(&tbl[v >> 1], 1u << sh) >> sh) & 0xFFFFu;
                } else {
                    uint32_t h = (v * 0x9E3779B1u) >> hshift;
                    for (int probe = 0; probe < words; ++probe) {
                        uint32_t cur = *reinterpret_cast<volatile uint32_t*>(tbl + h);
                        if (cur == kSlotEmpty) {
                            cur = atomicCAS(&tbl[h], kSlotEmpty, (v << 16) | 1u);
                            if (cur == kSlotEmpty) { rank = 0; break; }
                        }
                        if ((cur >> 16) == v) { rank = atomicAdd(&tbl[h], 1u) & 0xFFFFu; break; }
                        h = (h + 1u) & (uint32_t)(words - 1);
                    }
                }
            }
            const unsigned one = __ballot_sync(full, rank == 0u);
            if (rank == 0u) dst[nd + __popc(one & lt)] = (uint16_t)v;
            if (p0 == 0) first = __shfl_sync(full, v, __ffs(one) - 1);
            nd += __popc(one);
            const bool again = p < T && rank != 0u;
            const unsigned rep = __ballot_sync(full, again);
            if (again) {
                const int k = nr + __popc(rep & lt);
                if (k < kStaged) staged[k] = (rank << 16) | v;
            }
            nr += __popc(rep);
        }
        const int pad = (8 - (nd & 7)) & 7;
        if (lane < pad) dst[nd + lane] = (uint16_t)first;
        uint32_t at = 0;
        if (nr > 0) {
            if (lane == 0) at = atomicAdd(cursor, (uint32_t)nr);
            at = __shfl_sync(full, at, 0);
            __syncwarp();
            uint32_t done = at;
            if (nr <= kStaged)
                for (int q = lane; q < nr; q += 32) repeats[at + q] = staged[q];
            // more: every distinct K-mer's counter says how many it has
            for (int p0 = 0; p0 < nd && nr > kStaged; p0 += 32) {
                const int p = p0 + lane;
                uint32_t v = 0, c = 0;
                if (p < nd) {
                    v = *reinterpret_cast<volatile uint16_t*>(dst + p);
                    if (kDirect) {
                        c = (tbl[v >> 1] >> (16u * (v & 1u))) & 0xFFFFu;
                    } else {
                        uint32_t h = (v * 0x9E3779B1u) >> hshift;
                        for (int probe = 0; probe < words && (tbl[h] >> 16) != v; ++probe)
                            h = (h + 1u) & (uint32_t)(words - 1);
                        c = tbl[h] & 0xFFFFu;
                    }
                }
                const int extra = c > 1u ? (int)c - 1 : 0;
                int x = extra;
#pragma unroll
                for (int o = 1; o < 32; o <<= 1) {
                    const int y = __shfl_up_sync(full, x, o);
                    if (lane >= o) x += y;
                }
                for (int q = 0; q < extra; ++q) repeats[done + x - extra + q] = ((uint32_t)(q + 1) << 16) | v;
                done += __shfl_sync(full, x, 31);
            }
        }
        if (lane == 0) meta[i] = make_int4(nd, nr, (int)at, T);
        __syncwarp();
    }
}

// Per position the smallest count that can pass with it as the shorter read
// (smin), per 32 positions the smallest of these, and at K = 8 whether the
// read is H-heavy: |H| >= mmin[T], without which no pair of reads with
// different H keys can pass.
__global__ void filter_need_kernel(const int32_t* __restrict__ tcount, const uint16_t* __restrict__ smin,
                                   const uint16_t* __restrict__ mmin, const uint16_t* __restrict__ nh, int n,
                                   float* __restrict__ need, float* __restrict__ cmin,
                                   uint8_t* __restrict__ heavy, FilterCtl* ctl) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    float v = 1e9f;
    bool h = false;
    if (i < n) {
        const int T = tcount[i];
        const uint32_t s = smin[T];
        if (s != 0xFFFFu) v = (float)s;
        need[i] = v;
        if (nh != nullptr) {
            h = nh[i] >= mmin[T];
            heavy[i] = h;
        }
    }
    float c = v;
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) c = fminf(c, __shfl_xor_sync(0xffffffffu, c, o));
    if ((threadIdx.x & 31) == 0 && i < n) cmin[i >> 5] = c;
    if (nh != nullptr && __any_sync(0xffffffffu, h) && (threadIdx.x & 31) == 0) atomicOr(&ctl->any_heavy, 1u);
}

// K = 8: end of the run of equal H keys that holds a panel's last row.
__global__ void filter_panel_end_kernel(const uint32_t* __restrict__ hkey, int n, int panels,
                                        int32_t* __restrict__ pend) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= panels) return;
    const uint32_t key = hkey[min(n, 128 * p + 128) - 1];
    int lo = min(n, 128 * p + 128), hi = n;
    while (lo < hi) {
        const int mid = (lo + hi) / 2;
        if (hkey[mid] <= key) lo = mid + 1; else hi = mid;
    }
    pend[p] = lo;
}

// ---- the contraction --------------------------------------------------------

constexpr int kRows = 128;                 // row positions of a tile (TMEM lanes)
constexpr int kCols = 224;                 // column positions of a tile: two accumulators of
                                           // 224 columns leave 64 TMEM columns for the scales
constexpr int kChunkA = kRows * 128;       // 256 dimensions of a tile's rows (bytes)
constexpr int kChunkB = kCols * 128;
constexpr int kResidentChunks = 4;         // rows stay in shared memory up to 1,024 dimensions
constexpr int kMaxDepth = 3;               // stages of each of the two rings
constexpr int kCandBuf = 96;               // candidates a warp holds before it writes them out
constexpr int kEpilogueWarps = 12;         // for each quarter of the TMEM lanes:
constexpr int kEpiPer = kEpilogueWarps / 4;
constexpr int kEpiSteps = (kCols / 32 + kEpiPer - 1) / kEpiPer;
constexpr int kFilterThreads = 96 + 32 * kEpilogueWarps;   // warp 0 TMA, warps 1-2 MMA, then the epilogue
constexpr size_t kSmemLimit = 227 * 1024;
constexpr long long kWaitCycles = 4000000000ll;   // about two seconds

struct FilterArgs {
    const int4* items;    // (panel, first column tile, end column tile, -)
    const int2* segs;     // items of each segment: first, end
    int nsegs;
    int chunks;           // 256-dimension chunks of a signature
    int depth;            // stages of a ring
    int n;
    const float* need;
    const float* cmin;
    const uint16_t* excess;
    uint2* cand;          // (row, column)
    unsigned long long cap;
    int round;
    FilterCtl* ctl;
    long long wait;       // cycles a wait may take
};

struct Bars {
    uint64_t full[2 * kMaxDepth], empty[2 * kMaxDepth];
    uint64_t a_full, a_empty;
    uint64_t acc_full[2], acc_empty[2];
    uint64_t drain;
    uint32_t held[kEpilogueWarps];   // candidates in each warp's buffer
    uint32_t tmem;
    uint32_t abort;
};

__device__ __forceinline__ uint32_t smem_addr(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void bar_init(uint64_t* b, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_addr(b)), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_expect(uint64_t* b, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_addr(b)), "r"(bytes) : "memory");
}
__device__ __forceinline__ void bar_arrive(uint64_t* b) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_addr(b)) : "memory");
}
__device__ __forceinline__ bool bar_try(uint64_t* b, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(ok) : "r"(smem_addr(b)), "r"(parity) : "memory");
    return ok != 0;
}
// A wait that gives up after `limit` cycles (below 0: the loader's first one at
// once), or once another thread of the block has: the block then leaves its
// loops and the run reports a timeout.
struct Waiter {
    Bars* bars;
    FilterCtl* ctl;
    long long limit;
};
__device__ __noinline__ bool bar_wait_slow(uint64_t* b, uint32_t parity, const Waiter w) {
    const long long t0 = clock64();
    for (uint32_t i = 0;; ++i) {
        if ((i & 31u) == 0) {
            if (*reinterpret_cast<volatile uint32_t*>(&w.bars->abort)) return false;
            if (clock64() - t0 > w.limit) {
                *reinterpret_cast<volatile uint32_t*>(&w.bars->abort) = 1u;
                atomicOr(&w.ctl->timeout, 1u);
                return false;
            }
        }
        if (bar_try(b, parity)) return true;
    }
}
__device__ __forceinline__ bool bar_wait(uint64_t* b, uint32_t parity, const Waiter& w) {
    return (w.limit >= 0 && bar_try(b, parity)) || bar_wait_slow(b, parity, w);
}
// The same for a whole warp, which goes on or gives up as one: one lane's
// limit may run out as another's wait ends, and what follows a wait (elect,
// TMEM loads) needs all lanes.
__device__ __forceinline__ bool bar_wait_warp(uint64_t* b, uint32_t parity, const Waiter& w) {
    uint32_t all;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "vote.sync.all.pred p, p, 0xffffffff;\n"
        "selp.u32 %0, 1, 0, p;\n}"
        : "=r"(all) : "r"(smem_addr(b)), "r"(parity) : "memory");
    return all != 0 || __all_sync(0xffffffffu, bar_wait_slow(b, parity, w));
}

__device__ __forceinline__ void tma_load(const CUtensorMap* map, uint32_t dst, int x, int y, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
        ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(smem_addr(bar)) : "memory");
}
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "elect.sync _|p, 0xffffffff;\n"
        "selp.u32 %0, 1, 0, p;\n}" : "=r"(ok));
    return ok != 0;
}
// K-major operand, 128-byte swizzle: 8-row groups of 1,024 bytes.
__device__ __forceinline__ uint64_t operand_desc(uint32_t addr) {
    return (uint64_t)((addr & 0x3FFFFu) >> 4) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}

// e2m1 x e2m1, ue8m0 scales, M = 128, N = 224, FP32 accumulator.
constexpr uint32_t kInstr = (1u << 7) | (1u << 10) | ((uint32_t)(kCols >> 3) << 17) | (1u << 23) | (1u << 27);

__device__ __forceinline__ void mma_mxf4(uint32_t d, uint64_t a, uint64_t b, uint32_t sfa, uint32_t sfb,
                                         bool accumulate) {
    asm volatile(
        "{\n.reg .pred p;\n"
        "setp.ne.b32 p, %6, 0;\n"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%5], p;\n}"
        ::"r"(d), "l"(a), "l"(b), "r"(kInstr), "r"(sfa), "r"(sfb), "r"((uint32_t)accumulate) : "memory");
}
__device__ __forceinline__ void mma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];"
                 ::"r"(smem_addr(bar)) : "memory");
}

#define TMEM_LD32(v, addr)                                                                                   \
    asm volatile(                                                                                            \
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "                                                            \
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,"                                            \
        "%16,%17,%18,%19,%20,%21,%22,%23,%24,%25,%26,%27,%28,%29,%30,%31}, [%32];"                           \
        : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3]), "=f"(v[4]), "=f"(v[5]), "=f"(v[6]), "=f"(v[7]),    \
          "=f"(v[8]), "=f"(v[9]), "=f"(v[10]), "=f"(v[11]), "=f"(v[12]), "=f"(v[13]), "=f"(v[14]),           \
          "=f"(v[15]), "=f"(v[16]), "=f"(v[17]), "=f"(v[18]), "=f"(v[19]), "=f"(v[20]), "=f"(v[21]),         \
          "=f"(v[22]), "=f"(v[23]), "=f"(v[24]), "=f"(v[25]), "=f"(v[26]), "=f"(v[27]), "=f"(v[28]),         \
          "=f"(v[29]), "=f"(v[30]), "=f"(v[31])                                                              \
        : "r"(addr))

// Waits for the warp's TMEM loads; the values pass through, so that nothing
// reads them before the wait.
#define TMEM_WAIT32(v)                                                                                       \
    asm volatile("tcgen05.wait::ld.sync.aligned;"                                                            \
        : "+f"(v[0]), "+f"(v[1]), "+f"(v[2]), "+f"(v[3]), "+f"(v[4]), "+f"(v[5]), "+f"(v[6]), "+f"(v[7]),    \
          "+f"(v[8]), "+f"(v[9]), "+f"(v[10]), "+f"(v[11]), "+f"(v[12]), "+f"(v[13]), "+f"(v[14]),           \
          "+f"(v[15]), "+f"(v[16]), "+f"(v[17]), "+f"(v[18]), "+f"(v[19]), "+f"(v[20]), "+f"(v[21]),         \
          "+f"(v[22]), "+f"(v[23]), "+f"(v[24]), "+f"(v[25]), "+f"(v[26]), "+f"(v[27]), "+f"(v[28]),         \
          "+f"(v[29]), "+f"(v[30]), "+f"(v[31])                                                              \
        :: "memory")

__device__ __forceinline__ void tmem_fill32(uint32_t addr, uint32_t x) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1,%1};"
        ::"r"(addr), "r"(x) : "memory");
}

// Candidates of one warp: kept in shared memory, written out in runs.  Once
// one does not fit any more the warp takes no others (*stuffed): the pass has
// given up, and where every pair is a candidate taking them is most of its time.
__device__ __forceinline__ void cand_flush(const FilterArgs& a, const uint2* buf, int count, int lane, bool* stuffed) {
    if (count == 0) return;
    unsigned long long base = 0;
    if (lane == 0) base = atomicAdd(&a.ctl->cand[a.round], (unsigned long long)count);
    base = __shfl_sync(0xffffffffu, base, 0);
    for (int i = lane; i < count; i += 32)
        if (base + i < a.cap) a.cand[base + i] = buf[i];
    *stuffed = base + count > a.cap;
}

__device__ __forceinline__ float max3(float x, float y, float z) {
    float m;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(m) : "f"(x), "f"(y), "f"(z));
    return m;
}

// One 32 x 32 block of bounds: lane = row, v = 32 columns from c0 on.
__device__ __forceinline__ void take_candidates(const FilterArgs& a, const float (&v)[32], float thr, int row,
                                                int c0, uint2* buf, uint32_t* held, int lane, bool* stuffed) {
    if (*stuffed) return;
    float mx[4];
#pragma unroll
    for (int g = 0; g < 4; ++g) {
        mx[g] = max3(v[8 * g], v[8 * g + 1], v[8 * g + 2]);
        mx[g] = max3(mx[g], v[8 * g + 3], v[8 * g + 4]);
        mx[g] = max3(mx[g], v[8 * g + 5], fmaxf(v[8 * g + 6], v[8 * g + 7]));
    }
    const bool hit = fmaxf(max3(mx[0], mx[1], mx[2]), mx[3]) >= thr;
    if (!__any_sync(0xffffffffu, hit)) return;
    if (hit) {
        uint32_t mask = 0;
#pragma unroll
        for (int g = 0; g < 4; ++g) {
            if (mx[g] >= thr) {
#pragma unroll
                for (int e = 8 * g; e < 8 * g + 8; ++e) mask |= v[e] >= thr ? 1u << e : 0u;
            }
        }
        if (c0 + 32 > a.n) mask &= c0 < a.n ? (1u << (a.n - c0)) - 1u : 0u;
        const int d = row - c0;        // only columns beyond the row
        if (d >= 0) mask &= d >= 31 ? 0u : ~0u << (d + 1);
        const uint32_t mine = (uint32_t)__popc(mask);
        if (mine > 0) {
            const uint32_t at = atomicAdd(held, mine);
            unsigned long long out = 0;
            if (at + mine > (uint32_t)kCandBuf) {   // no room: the rest goes straight out
                const uint32_t room = at < (uint32_t)kCandBuf ? (uint32_t)kCandBuf - at : 0u;
                out = atomicAdd(&a.ctl->cand[a.round], (unsigned long long)(mine - room));
            }
            for (uint32_t k = at; mask; mask &= mask - 1, ++k) {
                const uint2 p = make_uint2((uint32_t)row, (uint32_t)(c0 + __ffs(mask) - 1));
                if (k < (uint32_t)kCandBuf) buf[k] = p;
                else if (out < a.cap) a.cand[out++] = p;
            }
        }
    }
    __syncwarp();
    const uint32_t n = *reinterpret_cast<volatile uint32_t*>(held);
    if (n > (uint32_t)kCandBuf / 2) {
        cand_flush(a, buf, (int)min(n, (uint32_t)kCandBuf), lane, stuffed);
        __syncwarp();
        if (lane == 0) *held = 0;
        __syncwarp();
    }
}

// One persistent block per SM.  All tiles, panel after panel, are cut into
// segments of equal length, and each block takes every so-many-th segment:
// the same number of tiles for everyone, from several places of the triangle
// (items of 64 tiles dealt in turn left the SMs idle for 14 % of the run).
// An item is 128 row positions (a panel) against a run of 224-column tiles.  The rows'
// signatures stay in shared memory for the whole item (up to 1,024
// dimensions; longer signatures stream rows and columns together), the
// columns' pass through two rings of 128-byte-wide TMA boxes, one for each
// of the two TMEM accumulators and its issuing warp, while twelve warps compare
// the other one with the rows' thresholds, 32 columns of 32 rows at a time.
// All block scales are 1.
//
// Bound: the 4-bit MMA rate (a 128 x 224 tile of 768 dimensions is 1,344
// cycles at 16,384 multiply-adds a cycle); the compare costs about 20
// instructions per 32 x 32 values unless one of them is a candidate.
// Measured, 99,999 reads of 300-500 nt at K = 6 (5.0e9 pairs, 768 dimensions,
// 2.70 M candidates): 1.25 ms, 0.59 of that rate (0.97 ms with the compares
// off, 1.87 ms with one issuing warp); the tile kernel took 7.26 ms.  Eight
// compare warps 1.32 ms, sixteen 1.24 ms.  20,000 reads: 67 us.  Blocks stand
// alone: pairs and fours that shared the columns' boxes took 1.24 and 1.56 ms
// (63-70 us for 20,000 reads).
template <bool kResident>
__global__ void __launch_bounds__(kFilterThreads, 1) kmer_filter_kernel(
    const __grid_constant__ CUtensorMap map_rows, const __grid_constant__ CUtensorMap map_cols, const FilterArgs a) {
    extern __shared__ uint8_t smem_raw[];
    const uint32_t smem0 = (smem_addr(smem_raw) + 1023u) & ~1023u;
    uint8_t* smem = smem_raw + (smem0 - smem_addr(smem_raw));
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int bytes_a = kResident ? a.chunks * kChunkA : 0;
    constexpr int kStage = kResident ? kChunkB : kChunkA + kChunkB;
    const uint32_t ring = smem0 + bytes_a;
    uint8_t* tail = smem + bytes_a + 2 * a.depth * kStage;
    uint2* cbuf = reinterpret_cast<uint2*>(tail);
    Bars* bars = reinterpret_cast<Bars*>(tail + kEpilogueWarps * kCandBuf * sizeof(uint2));
    const int first = (int)blockIdx.x, stride = (int)gridDim.x;
    // one thread looks: another block's wait may run out at any moment
    if (__syncthreads_or(threadIdx.x == 0 && pass_ended(a.ctl))) return;

    if (threadIdx.x == 0) {
        for (int s = 0; s < 2 * a.depth; ++s) { bar_init(&bars->full[s], 1); bar_init(&bars->empty[s], 1); }
        bar_init(&bars->a_full, 1);
        bar_init(&bars->a_empty, 2);
        for (int b = 0; b < 2; ++b) { bar_init(&bars->acc_full[b], 1); bar_init(&bars->acc_empty[b], kEpilogueWarps); }
        bar_init(&bars->drain, 2);
        for (int w = 0; w < kEpilogueWarps; ++w) bars->held[w] = 0;
        bars->abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 1) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;"
                     ::"r"(smem_addr(&bars->tmem)), "r"(512u) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    const uint32_t tmem = bars->tmem;
    const uint32_t scales = tmem + 2 * kCols;
    if (warp >= 3 && warp < 7) {
        // block scales: 2^0 everywhere (ue8m0 127)
        const uint32_t mine = scales + ((uint32_t)(32 * (warp & 3)) << 16);
        tmem_fill32(mine, 0x7F7F7F7Fu);
        tmem_fill32(mine + 32, 0x7F7F7F7Fu);
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");

    const Waiter wt{bars, a.ctl, a.wait};
    uint32_t steps[2] = {0, 0}, a_loads = 0;   // loads the loader has started
    if (warp == 0) {
        if (lane == 0) {
            // two rings of stages, for the even and the odd tiles: each ring
            // has one consumer, which meets every phase of its barriers
            uint32_t stage[2] = {0, 0}, phase[2] = {1, 1};
            uint32_t item = 0, tile = 0;
            const uint32_t depth = (uint32_t)a.depth;
            bool ok = true;
            for (int sg = first; sg < a.nsegs && ok; sg += stride)
            for (int it = __ldg(&a.segs[sg].x), end = __ldg(&a.segs[sg].y); it < end && ok; ++it, ++item) {
                const int4 q = __ldg(a.items + it);
                const int row0 = kRows * q.x;
                if (kResident) {
                    if (!bar_wait(&bars->a_empty, (item & 1) ^ 1, wt)) { ok = false; break; }
                    bar_expect(&bars->a_full, (uint32_t)bytes_a);
                    ++a_loads;
                    for (int k = 0; k < a.chunks; ++k)
                        tma_load(&map_rows, smem0 + k * kChunkA, 128 * k, row0, &bars->a_full);
                }
                for (int t = q.y; t < q.z && ok; ++t, ++tile) {
                    const uint32_t g = tile & 1u;
                    uint32_t st = stage[g], ph = phase[g];
                    for (int k = 0; k < a.chunks; ++k) {
                        const uint32_t slot = g * depth + st;
                        if (!bar_wait(&bars->empty[slot], ph, wt)) { ok = false; break; }
                        bar_expect(&bars->full[slot], kStage);
                        ++steps[g];
                        const uint32_t dst = ring + slot * kStage;
                        if (!kResident) tma_load(&map_rows, dst + kChunkB, 128 * k, row0, &bars->full[slot]);
                        tma_load(&map_cols, dst, 128 * k, kCols * t, &bars->full[slot]);
                        if (++st == depth) { st = 0; ph ^= 1; }
                    }
                    stage[g] = st;
                    phase[g] = ph;
                }
            }
            // the tensor cores' last arrivals, which no stage waits for: the
            // block's shared memory may be another's once it has ended
            for (uint32_t g = 0; g < 2 && ok; ++g)
                for (uint32_t s = 0; s < depth && ok; ++s) {
                    const uint32_t uses = steps[g] / depth + (s < steps[g] % depth ? 1u : 0u);
                    if (uses > 0) ok = bar_wait(&bars->empty[g * depth + s], (uses - 1) & 1, wt);
                }
            if (kResident && ok && item > 0) ok = bar_wait(&bars->a_empty, (item - 1) & 1, wt);
        }
        __syncwarp();
    } else if (warp <= 2) {
        // Two warps issue, one for each accumulator: an MMA costs its issuer
        // about 70 cycles and a chunk's barrier and commit as much again,
        // more than the 112 cycles it takes the tensor cores.  The whole warp
        // runs the loop, so that its operands stay in uniform registers; one
        // elected thread issues.
        const uint32_t mine = (uint32_t)warp - 1u;
        const uint32_t depth = (uint32_t)a.depth, slot0 = mine * depth;
        uint32_t stage = 0, phase = 0, item = 0, tile = 0, bphase = 1;
        bool ok = true;
        const uint64_t desc_a = operand_desc(smem0), desc_b = operand_desc(ring + slot0 * kStage);
        const uint32_t acc = tmem + mine * kCols;
        for (int sg = first; sg < a.nsegs && ok; sg += stride)
        for (int it = __ldg(&a.segs[sg].x), end = __ldg(&a.segs[sg].y); it < end && ok; ++it, ++item) {
            const int4 q = __ldg(a.items + it);
            if (kResident && !bar_wait_warp(&bars->a_full, item & 1, wt)) { ok = false; break; }
            for (int t = q.y; t < q.z && ok; ++t, ++tile) {
                if ((tile & 1u) != mine) continue;
                if (!bar_wait_warp(&bars->acc_empty[mine], bphase, wt)) { ok = false; break; }
                bphase ^= 1;
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                for (int k = 0; k < a.chunks; ++k) {
                    if (!bar_wait_warp(&bars->full[slot0 + stage], phase, wt)) { ok = false; break; }
                    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                    const uint64_t db = desc_b + stage * (kStage >> 4);
                    const uint64_t da = kResident ? desc_a + k * (kChunkA >> 4) : db + (kChunkB >> 4);
                    if (elect_one()) {
#pragma unroll
                        for (int i = 0; i < 4; ++i)   // 64 dimensions (32 bytes) each
                            mma_mxf4(acc, da + 2 * i, db + 2 * i, scales, scales + 32, k + i > 0);
                        mma_commit(&bars->empty[slot0 + stage]);
                        if (k == a.chunks - 1) mma_commit(&bars->acc_full[mine]);
                    }
                    __syncwarp();
                    if (++stage == depth) { stage = 0; phase ^= 1; }
                }
            }
            if (ok && kResident && elect_one()) mma_commit(&bars->a_empty);
            __syncwarp();
        }
        __syncwarp();
    } else {
        const int part = warp & 3;                     // TMEM lanes 32 part .. 32 part + 31
        const int lead = (warp - 3) >> 2;              // its first 32-column step
        uint2* mine = cbuf + (warp - 3) * kCandBuf;
        uint32_t* held = &bars->held[warp - 3];
        uint32_t tile = 0;
        bool ok = true, stuffed = false;
        for (int sg = first; sg < a.nsegs && ok; sg += stride)
        for (int it = __ldg(&a.segs[sg].x), end = __ldg(&a.segs[sg].y); it < end && ok; ++it) {
            const int4 q = __ldg(a.items + it);
            const int row = kRows * q.x + 32 * part + lane;
            const float rneed = row < a.n ? __ldg(a.need + row) : 1e9f;
            // half a count of slack: S is a multiple of 1/4
            const float rx = row < a.n ? (float)__ldg(a.excess + row) + 0.5f : 0.0f;
            for (int t = q.y; t < q.z; ++t, ++tile) {
                const uint32_t b = tile & 1, use = tile >> 1;
                const int c0 = kCols * t + 32 * lead;      // this warp's columns: 32 of every 32 kEpiPer
                float need[kEpiSteps];
#pragma unroll
                for (int k = 0; k < kEpiSteps; ++k) {
                    const int c = c0 + 32 * kEpiPer * k;
                    need[k] = c < a.n && row < a.n ? fminf(rneed, __ldg(a.cmin + (c >> 5))) - rx : 1e9f;
                }
                if (!bar_wait_warp(&bars->acc_full[b], use & 1, wt)) { ok = false; break; }
                asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
                const uint32_t acc = tmem + b * kCols + 32 * lead + ((uint32_t)(32 * part) << 16);
                // one block of 32 columns on its way while the other is compared
                float v[2][32];
                TMEM_LD32(v[0], acc);
#pragma unroll
                for (int k = 0; k < kEpiSteps; ++k) {
                    if (kEpiPer * k + lead < kCols / 32) {
                        TMEM_WAIT32(v[k & 1]);
                        if (kEpiPer * (k + 1) + lead < kCols / 32) {
                            TMEM_LD32(v[(k + 1) & 1], acc + 32 * kEpiPer * (k + 1));
                        } else {
                            // the accumulator is free before the last compare
                            asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
                            __syncwarp();
                            if (lane == 0) bar_arrive(&bars->acc_empty[b]);
                        }
                        take_candidates(a, v[k & 1], need[k], row, c0 + 32 * kEpiPer * k, mine, held, lane, &stuffed);
                    }
                }
            }
        }
        __syncwarp();
        cand_flush(a, mine, (int)min(*reinterpret_cast<volatile uint32_t*>(held), (uint32_t)kCandBuf), lane, &stuffed);
    }
    __syncthreads();   // every warp has left its loops
    if (*reinterpret_cast<volatile uint32_t*>(&bars->abort)) {
        // the block gives up: let its copies land and its MMAs end first
        const long long t0 = clock64();
        if (threadIdx.x == 0) {
            for (uint32_t g = 0; g < 2; ++g)
                for (uint32_t s = 0; s < (uint32_t)a.depth; ++s) {
                    const uint32_t uses = steps[g] / a.depth + (s < steps[g] % a.depth ? 1u : 0u);
                    while (uses > 0 && !bar_try(&bars->full[g * a.depth + s], (uses - 1) & 1) &&
                           clock64() - t0 < kWaitCycles) {}
                }
            while (a_loads > 0 && !bar_try(&bars->a_full, (a_loads - 1) & 1) && clock64() - t0 < kWaitCycles) {}
        } else if (warp == 1 || warp == 2) {
            if (elect_one()) mma_commit(&bars->drain);   // two arrivals
            __syncwarp();
            while (!bar_try(&bars->drain, 0) && clock64() - t0 < kWaitCycles) {}
            __syncwarp();
        }
    }
    asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory");
    if (warp == 1)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512u));
}

// ---- the exact count --------------------------------------------------------

struct VerifyArgs {
    const uint2* cand;
    uint32_t* candidx;        // index of a candidate among its row's
    uint2* sorted;            // (row, column), the candidates of a row together
    uint32_t* rowcnt;
    uint32_t* rowoff;
    unsigned long long cap;
    const uint32_t* repeated; // repeats of all reads
    float tuples;             // tuples of all reads
    double most;              // candidates worth counting, were none dearer than usual
    int round;
    FilterCtl* ctl;
    const uint16_t* distinct;
    int dstride;
    const int4* meta;         // per position: distinct K-mers, repeats, first repeat, tuples
    const uint32_t* repeats;
    const int32_t* perm;      // position -> read ID (K = 8), nullptr: identity
    const uint32_t* hkey;     // K = 8
    const uint8_t* heavy;     // K = 8
    const uint16_t* mmin;
    int n, K, rep_slots;
    int olo, ohi;
    int A, sd;
    unsigned long long* counter;
    uint64_t* keys;
    uint32_t* vals;
    int64_t out_cap;
};

// True when the round's candidates are there, fit and are worth counting: a
// candidate costs more where most of a read's K-mers are repeats (reads of few
// bases: 1.7 ns for 0.3 with 0.88 of them; 0.06 to 0.28 are usual).
__device__ __forceinline__ bool round_fits(const VerifyArgs& a, unsigned long long found) {
    if (pass_ended(a.ctl)) return false;
    const float dearer = 1.0f + 8.0f * fmaxf(0.0f, (float)*a.repeated / a.tuples - 0.3f);
    if (found <= a.cap && (dearer == 1.0f || (double)found * dearer <= a.most)) return true;
    if (blockIdx.x == 0 && threadIdx.x == 0) atomicOr(&a.ctl->overflow, 1u);
    return false;
}

// Candidates per row, and each one's index among its row's.
__global__ void __launch_bounds__(256) filter_count_kernel(const VerifyArgs a) {
    const unsigned long long found = a.ctl->cand[a.round];
    if (!round_fits(a, found)) return;
    for (unsigned long long i = (unsigned long long)blockIdx.x * 256 + threadIdx.x; i < found; i += gridDim.x * 256ull)
        a.candidx[i] = atomicAdd(a.rowcnt + a.cand[i].x, 1u);
}

// A stretch of the sorted list for each row with candidates (rows in any
// order: one atomic per warp); clears the counts for the next round.
__global__ void __launch_bounds__(256) filter_rows_kernel(const VerifyArgs a) {
    if (!round_fits(a, a.ctl->cand[a.round])) return;
    const int r = blockIdx.x * 256 + threadIdx.x;
    const int lane = threadIdx.x & 31;
    const uint32_t c = r < a.n ? a.rowcnt[r] : 0u;
    uint32_t x = c;
#pragma unroll
    for (int o = 1; o < 32; o <<= 1) {
        const uint32_t y = __shfl_up_sync(0xffffffffu, x, o);
        if (lane >= o) x += y;
    }
    uint32_t base = 0;
    if (lane == 31 && x > 0) base = atomicAdd(&a.ctl->cursor[a.round], x);
    base = __shfl_sync(0xffffffffu, base, 31);
    if (r < a.n && c > 0) {
        a.rowoff[r] = base + x - c;
        a.rowcnt[r] = 0;
    }
}

__global__ void __launch_bounds__(256) filter_scatter_kernel(const VerifyArgs a) {
    const unsigned long long found = a.ctl->cand[a.round];
    if (!round_fits(a, found)) return;
    for (unsigned long long i = (unsigned long long)blockIdx.x * 256 + threadIdx.x; i < found; i += gridDim.x * 256ull) {
        const uint2 p = a.cand[i];
        a.sorted[a.rowoff[p.x] + a.candidx[i]] = p;
    }
}

constexpr int kVerifyWarps = 8;

// Slots of the table of a row's repeats, filled to a half at the most: five
// times the repeats that a read of max_t random K-mers has (21 of 394 at K = 6,
// 213 of 1,400), since reads are not random.  Rows with more (few bases over and
// over) fill it part by part.
int rep_slots_for(int k, int max_t) {
    const double kinds = (double)(1 << (2 * k));
    const double repeats = max_t - kinds * (1.0 - std::exp(-max_t / kinds));
    int slots = 256;
    while (slots < 1024 && slots < 5.0 * repeats) slots *= 2;
    return slots;
}

// A warp takes up to 32 consecutive candidates of the sorted list.  Per row
// (about 4 to 30 candidates each) it marks the row's distinct K-mers in a map
// in shared memory -- a byte each for short reads up to K = 6 (4 KB a warp; a
// look-up is one load and one add), a bit each otherwise -- and puts its repeats in a small
// table; per candidate it streams the column's lists, eight K-mers to a
// 128-bit load, and looks each K-mer up.  The first words of the next
// candidate are on their way while one is counted.  The map is cleared
// through the row's list, so its size costs nothing per row.
//
// Bound: the look-ups' shared-memory wavefronts (about 3 per 32 random
// addresses) and issue slots.  2.70 M candidates of 400 nt: 0.88 ms (1.3 ms
// with every repeat looked up and bit marks; 8.5 ms with a hash table per
// pair and no grouping by row).
template <bool kBytes, bool kK8>
__global__ void __launch_bounds__(kVerifyWarps * 32, kK8 ? 3 : 5) filter_verify_kernel(const VerifyArgs a) {
    extern __shared__ __align__(16) uint32_t vsmem[];
    const unsigned full = 0xffffffffu;
    const unsigned long long found = a.ctl->cand[a.round];
    if (!round_fits(a, found)) return;
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int mwords = kBytes ? 1 << (2 * a.K - 2) : 1 << (2 * a.K - 5);
    const uint32_t rmask = (uint32_t)a.rep_slots - 1u;
    const int rshift = __clz(a.rep_slots) + 1;      // 32 - log2(slots)
    const int rep_most = a.rep_slots / 2;
    uint32_t* map = vsmem + warp * (mwords + a.rep_slots);
    uint8_t* mapb = reinterpret_cast<uint8_t*>(map);
    uint32_t* rt = map + mwords;
    for (int q = lane; q < mwords; q += 32) map[q] = 0;
    for (int q = lane; q < a.rep_slots; q += 32) rt[q] = kSlotEmpty;
    __syncwarp();
    // the marks of a row's list set or taken back
    auto mark = [&](const uint4* list, int nd, bool on) {
        for (int q = lane; q < (nd + 7) / 8; q += 32) {
            const uint4 e = list[q];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t w = k == 0 ? e.x : k == 1 ? e.y : k == 2 ? e.z : e.w;
                if (kBytes) {
                    mapb[w & 0xFFFFu] = on;
                    mapb[w >> 16] = on;
                } else if (on) {
                    atomicOr(&map[(w & 0xFFFFu) >> 5], 1u << (w & 31u));
                    atomicOr(&map[w >> 21], 1u << ((w >> 16) & 31u));
                } else {
                    map[(w & 0xFFFFu) >> 5] = 0;
                    map[w >> 21] = 0;
                }
            }
        }
    };
    auto put_repeats = [&](int first, int count) {
        for (int q = lane; q < count; q += 32) {
            const uint32_t e = a.repeats[first + q];
            uint32_t h = (e * 0x9E3779B1u) >> rshift;
            while (atomicCAS(&rt[h], kSlotEmpty, e) != kSlotEmpty) h = (h + 1u) & rmask;
        }
    };
    const int64_t total = (int64_t)found;
    const int64_t nw = (int64_t)gridDim.x * kVerifyWarps;
    const int batch = (int)min((int64_t)32, (total + nw - 1) / nw);
    int cur = -1;
    int4 mr = make_int4(0, 0, 0, 0);
    for (int64_t b0 = ((int64_t)blockIdx.x * kVerifyWarps + warp) * batch; b0 < total; b0 += nw * batch) {
        const int cnt = (int)min((int64_t)batch, total - b0);
        uint2 rc = make_uint2(0u, 0u);
        uint32_t sizes = 0, first_rep = 0;     // distinct K-mers | repeats << 16; first repeat
        uint32_t lim = 0xFFFFu;                // smallest count that passes
        bool same = true, live = false;
        if (lane < cnt) {
            rc = a.sorted[b0 + lane];
            const int4 m = a.meta[rc.y];
            sizes = (uint32_t)m.x | (uint32_t)m.y << 16;
            first_rep = (uint32_t)m.z;
            lim = a.mmin[min(m.w, a.meta[rc.x].w)];
            live = lim != 0xFFFFu;
            if (kK8) {
                // reads of different H keys share no L half, and can pass
                // only with an H-heavy read among them
                same = a.hkey[rc.x] == a.hkey[rc.y];
                live = live && (same || (a.heavy[rc.x] | a.heavy[rc.y]) != 0);
            }
        }
        int my_m = 0, my_mn = 0;
        unsigned todo = __ballot_sync(full, live);
        int i = todo ? __ffs(todo) - 1 : 0;
        uint32_t c = __shfl_sync(full, rc.y, i), sz = __shfl_sync(full, sizes, i);
        uint4 head = make_uint4(0u, 0u, 0u, 0u);
        if (kBytes && todo && 8 * lane < (int)(sz & 0xFFFFu))
            head = reinterpret_cast<const uint4*>(a.distinct + (int64_t)c * a.dstride)[lane];
        while (todo) {
            todo &= todo - 1;
            // the next candidate
            const int i2 = todo ? __ffs(todo) - 1 : i;
            const uint32_t c2 = __shfl_sync(full, rc.y, i2), sz2 = __shfl_sync(full, sizes, i2);
            uint4 head2 = head;
            if (kBytes && todo && 8 * lane < (int)(sz2 & 0xFFFFu))
                head2 = reinterpret_cast<const uint4*>(a.distinct + (int64_t)c2 * a.dstride)[lane];
            const int r = (int)__shfl_sync(full, rc.x, i);
            if (r != cur) {
                if (cur >= 0) {
                    mark(reinterpret_cast<const uint4*>(a.distinct + (int64_t)cur * a.dstride), mr.x, false);
                    if (mr.y > 0) for (int q = lane; q < a.rep_slots; q += 32) rt[q] = kSlotEmpty;
                    __syncwarp();
                }
                cur = r;
                mr = a.meta[r];
                mark(reinterpret_cast<const uint4*>(a.distinct + (int64_t)r * a.dstride), mr.x, true);
                if (mr.y <= rep_most) put_repeats(mr.z, mr.y);
                __syncwarp();
            }
            const int nd = (int)(sz & 0xFFFFu), nr = (int)(sz >> 16);
            // K = 8, different keys: only the K-mers >= 0x8000 (H) count
            const bool both = !kK8 || __shfl_sync(full, (int)same, i) != 0;
            const int nq = (nd + 7) / 8;
            uint32_t m = 0;
            for (int q = lane; q < nq; q += 32) {
                const uint4 e = kBytes && q == lane ? head
                                                    : reinterpret_cast<const uint4*>(a.distinct + (int64_t)c * a.dstride)[q];
                uint32_t hits = 0, first = 0;
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const uint32_t w = k == 0 ? e.x : k == 1 ? e.y : k == 2 ? e.z : e.w;
                    uint32_t lo, hi;
                    if (kBytes) {
                        lo = mapb[w & 0xFFFFu];
                        hi = mapb[w >> 16];
                    } else {
                        lo = (map[(w & 0xFFFFu) >> 5] >> (w & 31u)) & 1u;
                        hi = (map[w >> 21] >> ((w >> 16) & 31u)) & 1u;
                    }
                    if (!both) {
                        lo &= w >> 15;
                        hi &= w >> 31;
                    }
                    if (k == 0) first = lo;
                    hits += lo + hi;
                }
                m += hits;
                // the padding: copies of the list's first K-mer
                if (q == 0) m -= first * (uint32_t)(8 * nq - nd);
            }
            // the repeats only where they can still lift the count over the cut
            m = __reduce_add_sync(full, m);
            if (nr > 0 && m + (uint32_t)min(nr, mr.y) >= __shfl_sync(full, lim, i)) {
                const uint32_t rep = __shfl_sync(full, first_rep, i);
                uint32_t more = 0;
                // a row with more repeats than the table takes at once fills it
                // part by part
                for (int k0 = 0; k0 < mr.y; k0 += rep_most) {
                    if (mr.y > rep_most) {
                        __syncwarp();
                        for (int q = lane; q < a.rep_slots; q += 32) rt[q] = kSlotEmpty;
                        __syncwarp();
                        put_repeats(mr.z + k0, min(rep_most, mr.y - k0));
                        __syncwarp();
                    }
                    for (int q = lane; q < nr; q += 32) {
                        const uint32_t e = a.repeats[rep + q];
                        if (!both && !(e & 0x8000u)) continue;
                        uint32_t h = (e * 0x9E3779B1u) >> rshift;
                        uint32_t v;
                        while ((v = rt[h]) != kSlotEmpty && v != e) h = (h + 1u) & rmask;
                        more += v == e;
                    }
                }
                m += __reduce_add_sync(full, more);
            }
            if (lane == i) {
                my_m = (int)m;
                my_mn = min(mr.w, nd + nr);
            }
            i = i2;
            c = c2;
            sz = sz2;
            head = head2;
        }
        bool pass = false;
        if (live) {
            pass = (uint32_t)my_m >= lim;
            if (a.perm == nullptr) pass = pass && (int)rc.x >= a.olo && (int)rc.x < a.ohi;
        }
        emit(a.counter, a.keys, a.vals, a.out_cap, a.A, a.sd, a.perm, a.olo, a.ohi, pass, (int)rc.x,
             (int)rc.y, my_m, my_mn);
    }
}

// ---- host side --------------------------------------------------------------

using EncodeFn = CUresult (*)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*,
                              const cuuint64_t*, const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave,
                              CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

EncodeFn tensor_map_encode() {
    static EncodeFn fn = [] {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult st;
        if (cudaGetDriverEntryPointByVersion("cuTensorMapEncodeTiled", &p, 12000, cudaEnableDefault, &st) != cudaSuccess) p = nullptr;
        return reinterpret_cast<EncodeFn>(p);
    }();
    return fn;
}

// Signatures as rows of bytes; a box is 128 bytes (256 dimensions) of
// `rows` positions.  Positions past the end read as zero.
int signature_map(crispy_ctx* ctx, CUtensorMap* map, void* sig, int row_bytes, int n, int rows) {
    EncodeFn enc = tensor_map_encode();
    if (!enc) return fail(ctx, CRISPY_E_DEVICE, "cuTensorMapEncodeTiled is not available");
    const cuuint64_t dims[2] = {(cuuint64_t)row_bytes, (cuuint64_t)n};
    const cuuint64_t strides[1] = {(cuuint64_t)row_bytes};
    const cuuint32_t box[2] = {128u, (cuuint32_t)rows};
    const cuuint32_t step[2] = {1u, 1u};
    const CUresult r = enc(map, CU_TENSOR_MAP_DATA_TYPE_UINT8, 2, sig, dims, strides, box, step,
                           CU_TENSOR_MAP_INTERLEAVE_NONE, CU_TENSOR_MAP_SWIZZLE_128B,
                           CU_TENSOR_MAP_L2_PROMOTION_L2_256B, CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) return fail(ctx, CRISPY_E_DEVICE, "cuTensorMapEncodeTiled failed (%d)", (int)r);
    return CRISPY_OK;
}

int log2_bits(uint64_t v) {
    int b = 0;
    while (b < 64 && (v >> b) != 0) ++b;
    return b;
}

}  // namespace

namespace {
// Candidates a round may leave: 1/256 of its pairs and 3.1 M at K = 6, less
// where the tile kernels are faster (K = 7 and 8) or a candidate dearer (K = 5:
// more repeats).  Beyond that (one OTU holds a good part of the reads) counting
// one by one costs more than the tile kernels.  Both cost the same at about
// 3.9 M candidates for 20,000 reads of 250 nt, 9 M for 50,000, 4.2 M for 12,000
// of 300-500 nt, 23 M for 100,000, 2.9 M for 11,000 at K = 5, 2.4 M for 12,000
// and 6 M for 30,000 at K = 7, 1.8 M for 20,000 of 250 nt at K = 8.  Whole
// kmerDist calls, filter against tiles: 20,000 reads in Zipf's proportions
// (4.0 M) 1,543 and 1,888 us, three tenths of them in one OTU (8.1 M) 2,864 and
// 2,110; 100,000 with 0.07 in one (15 M) 8.0 and 10.6 ms, with 0.15 (54 M) 22.0
// and 13.2.  (CRISPY_KMER_CAND sets the room, for tests: N, or below 0 one in -N of
// the pairs.)
int64_t candidates_worth(int64_t pairs, int k) {
    if (const char* e = std::getenv("CRISPY_KMER_CAND")) {
        const int64_t v = std::atoll(e);
        return std::max<int64_t>(1, v < 0 ? pairs / -v : v);
    }
    const int64_t base = (int64_t)(k <= 5 ? 11 : k == 6 ? 12 : k == 7 ? 9 : 6) << 18;
    return std::min<int64_t>(1 << 25, pairs / 256 + base);
}
int64_t candidate_room(int64_t pairs, int k) {
    return std::min<int64_t>(candidates_worth(pairs, k), std::max<int64_t>(pairs, 1));
}

// Their buffer: a quarter more, so that a set which the probe lets pass by a
// little does not fail at the end after all.
int64_t candidate_buffer(int64_t room) { return room + room / 4; }

// The probe: before the rest, one short run of tiles for each block, spread
// evenly over all of them (it is the run's first work, none of it twice).  If
// its candidates say that the room will not do, everything behind it ends at
// once, the exact lists included, and the tile kernels take the reads.  Sets
// of fewer tiles than this for each block are bounded without one: the whole
// contraction takes no longer than the rest of the attempt.
constexpr int64_t kProbeFrom = 16;

// Bins of the fold, in chunks of 256: two per K-mer of a mean read for tight
// cuts, three for loose ones.  Share of the pairs left as candidates, over
// the share that survives (reads of 250, 400 and 1,400 nt, K = 5..8): at
// 2 T bins 2 to 5 times at cuts up to 0.15 but 4 to 12 times at 0.3, at 3 T
// bins 1.5 to 4 times at 0.3; 1.3 T bins leave 6 to 15 times at 0.12.
constexpr float kMostCut = 0.3f;
int dims_wanted(int64_t tuples, int n, float thr) {
    const int mean = (int)(tuples / std::max(1, n));
    const int halves = thr <= 0.15f ? 4 : thr <= 0.25f ? 5 : 6;
    return halves * mean / 2;
}
int dims_for(int64_t tuples, int n, int k, float thr) {
    const int most = std::min(1 << (2 * k), 4096);
    return std::min(most, std::max(1, (dims_wanted(tuples, n, thr) + 128) / 256) * 256);
}
// Whether 4^K bins are enough of those (K = 5 has 1,024): kmerDist calls,
// filter against tiles, at 2.0 times as many wanted 1,073 and 2,256 us (15,000
// reads of 1,000 nt, cut 0.05) but 2,418 and 1,954 (6,000, cut 0.15), at 1.7
// times 1,118 and 1,704 (6,000 of 850 nt, cut 0.15) but 2,478 and 1,456 (6,000
// of 600 nt, cut 0.3), at 1.5 times 1,338 and 1,363 (6,000 of 500 nt, cut 0.3).
bool dims_do(int64_t tuples, int n, int k, float thr) {
    const float most = thr <= 0.08f ? 2.0f : thr <= 0.15f ? 1.7f : 1.5f;
    return (float)dims_wanted(tuples, n, thr) <= most * (float)std::min(1 << (2 * k), 4096);
}
}  // namespace

// Device bytes the filter's buffers take for reads of these lengths (and
// genDist's copy of the packed reads).
size_t kmer_filter_bytes(const int32_t* len, int n, int k) {
    if (k < 5 || n <= 0) return 0;
    int64_t tuples = 0, most = 0, max_len = 0;
    for (int r = 0; r < n; ++r) {
        const int64_t t = std::max(0, len[r] - k + 1);
        tuples += t;
        most = std::max(most, t);
        max_len = std::max<int64_t>(max_len, len[r]);
    }
    const int64_t read = 2 * (max_len / 16 + 5) * 4 + dims_for(tuples, n, k, kMostCut) / 2 + (most + 8) * 2 + 64;
    const int64_t pairs = (int64_t)n * (n + 512) / 2;
    return (size_t)(n * read + tuples * 4 + candidate_buffer(candidate_room(pairs, k)) * 20 + pairs / (kRows * kCols) * 16 + (1 << 20));
}

// Rule: K >= 5 (K = 4 has 256 bins at most, and the bound leaves a third to
// all of the pairs) and a cut of at most 0.3 (at 0.35 and above 7-30 % of
// the pairs stay at K = 5, and counting those one by one costs more than the
// tile kernels), with bins enough for the reads' length.  CRISPY_KMER_FILTER=0 turns
// it off; so do the variables that pick the tile kernels' own forms.  Reads
// that gave it up once do so at every cut as loose while they stay prepared.
bool kmer_filter_applies(const KmerJob& j, float thr) {
    if (j.k < 5 || !(thr <= kMostCut) || j.max_t < 1 || thr >= j.f_gave_up) return false;
    if (!dims_do(j.sum_t, j.n, j.k, thr)) return false;
    const char* e = std::getenv("CRISPY_KMER_FILTER");
    if (e && e[0] == '0') return false;
    for (const char* v : {"CRISPY_KMER_SPLIT", "CRISPY_KMER_QFIRE", "CRISPY_KMER_PREP_WARP",
                          "CRISPY_KMER_K8_SPLIT", "CRISPY_KMER_K8_QUEUE"})
        if (std::getenv(v)) return false;
    return true;
}

// Packed reads, K = 8 read order, fold and signatures of the prepared reads;
// their exact lists come with the first pass that needs them.
int kmer_filter_build(crispy_ctx* ctx, float thr) {
    KmerJob& j = ctx->kmer;
    cudaStream_t s = ctx->stream;
    const int n = j.n, k = j.k;
    const int K4 = 1 << (2 * k);
    const int64_t tuples = j.sum_t;
    const int dims = dims_for(tuples, n, k, thr);
    if (j.f_ready && j.f_dims == dims) return CRISPY_OK;
    j.f_ready = j.f_lists = false;
    j.f_dims = dims;
    j.f_stride = ((j.max_len + 15) / 16 + 1 + 3) / 4 * 4;
    j.f_dstride = (j.max_t + 7) / 8 * 8;
    CRISPY_TRY(ensure(ctx, j.f_packed, (size_t)n * j.f_stride * 4));
    CRISPY_TRY(ensure(ctx, j.f_hist, (size_t)K4 * 4 + 16));   // and the repeats' cursor
    CRISPY_TRY(ensure(ctx, j.f_map, (size_t)K4 * 2));
    CRISPY_TRY(ensure(ctx, j.f_sig, (size_t)n * (j.f_dims / 2)));
    CRISPY_TRY(ensure(ctx, j.f_excess, (size_t)n * 2));
    CRISPY_TRY(ensure(ctx, j.f_distinct, (size_t)n * j.f_dstride * 2));
    CRISPY_TRY(ensure(ctx, j.f_meta, (size_t)n * sizeof(int4)));
    CRISPY_TRY(ensure(ctx, j.f_repeats, (size_t)std::max<int64_t>(tuples, 1) * 4));
    uint64_t* keys = nullptr;
    uint32_t* idx = nullptr;
    const int tbits = std::max(1, log2_bits((uint64_t)j.max_t));
    if (k == 8) {
        CRISPY_TRY(ensure(ctx, j.keys, (size_t)n * 8));
        CRISPY_TRY(ensure(ctx, j.keys_alt, (size_t)n * 8));
        CRISPY_TRY(ensure(ctx, j.vals, (size_t)n * 4));
        CRISPY_TRY(ensure(ctx, j.vals_alt, (size_t)n * 4));
        CRISPY_TRY(ensure(ctx, j.sort_tmp, sort_tmp_bytes(n)));
        CRISPY_TRY(ensure(ctx, j.f_perm, (size_t)n * 4));
        CRISPY_TRY(ensure(ctx, j.f_t, (size_t)n * 4));
        CRISPY_TRY(ensure(ctx, j.f_hkey, (size_t)n * 4));
        CRISPY_TRY(ensure(ctx, j.f_nh, (size_t)n * 2));
        keys = j.keys.as<uint64_t>();
        idx = j.vals.as<uint32_t>();
    }
    const int grid = std::min((n + kPackWarps - 1) / kPackWarps, ctx->sm_count * 8);
    filter_pack_kernel<<<grid, kPackWarps * 32, 0, s>>>(j.seq.as<uint8_t>(), j.off.as<int64_t>(),
                                                       j.t0.as<int32_t>(), n, k, j.f_stride,
                                                       j.f_packed.as<uint32_t>(), tbits, keys, idx);
    count_launch(ctx);
    const int32_t* t = j.t0.as<int32_t>();
    const int32_t* perm = nullptr;
    if (k == 8) {
        uint64_t* sk = nullptr;
        uint32_t* sv = nullptr;
        CRISPY_TRY(sort_u64_payload(ctx, s, keys, j.keys_alt.as<uint64_t>(), idx, j.vals_alt.as<uint32_t>(), n,
                                    32 + tbits, true, &sk, &sv, j.sort_tmp));
        filter_order_kernel<<<(n + 255) / 256, 256, 0, s>>>(sk, sv, n, tbits, j.f_perm.as<int32_t>(),
                                                            j.f_t.as<int32_t>(), j.f_hkey.as<uint32_t>());
        count_launch(ctx);
        t = j.f_t.as<int32_t>();
        perm = j.f_perm.as<int32_t>();
    }
    CRISPY_CK(ctx, cudaMemsetAsync(j.f_hist.ptr, 0, (size_t)K4 * 4 + 16, s));
    const int sample = std::min(n, 1024);
    filter_hist_kernel<<<(sample + 7) / 8, 256, 0, s>>>(j.f_packed.as<uint32_t>(), j.f_stride,
                                                        j.t0.as<int32_t>(), n, k, sample, j.f_hist.as<uint32_t>());
    filter_map_kernel<<<1, 1024, 0, s>>>(j.f_hist.as<uint32_t>(), K4, j.f_dims, j.f_map.as<uint16_t>());
    const size_t smem = (size_t)kSigWarps * j.f_dims * 2;
    CRISPY_TRY(open_smem(ctx, filter_sig_kernel));
    filter_sig_kernel<<<std::min((n + kSigWarps - 1) / kSigWarps, ctx->sm_count * 8), kSigWarps * 32, smem, s>>>(
        j.f_packed.as<uint32_t>(), j.f_stride, t, perm, n, k, j.f_dims, j.f_map.as<uint16_t>(),
        j.f_sig.as<uint32_t>(), j.f_excess.as<uint16_t>(), k == 8 ? j.f_nh.as<uint16_t>() : nullptr);
    count_launch(ctx, 3);
    CRISPY_CK(ctx, cudaGetLastError());
    j.f_ready = true;
    return CRISPY_OK;
}

namespace {
// The exact lists of the prepared reads, unless the pass has ended by then.
int build_lists(crispy_ctx* ctx, FilterCtl* ctl, unsigned long long most) {
    KmerJob& j = ctx->kmer;
    cudaStream_t s = ctx->stream;
    const int n = j.n, k = j.k;
    const int K4 = 1 << (2 * k);
    const int32_t* t = k == 8 ? j.f_t.as<int32_t>() : j.t0.as<int32_t>();
    const int32_t* perm = k == 8 ? j.f_perm.as<int32_t>() : nullptr;
    // (a pass that gave up or ran out of time may have built them already)
    CRISPY_CK(ctx, cudaMemsetAsync(j.f_hist.as<uint32_t>() + K4, 0, 4, s));
    const bool direct = k <= 6;
    const int slots_log2 = j.max_t <= 512 ? 10 : j.max_t <= 1024 ? 11 : 12;
    const int words = direct ? K4 / 2 : 1 << slots_log2;
    const size_t lsmem = (size_t)kListWarps * words * 4;
    auto lists = direct ? filter_lists_kernel<true> : filter_lists_kernel<false>;
    CRISPY_TRY(open_smem(ctx, lists));
    lists<<<std::min((n + kListWarps - 1) / kListWarps, ctx->sm_count * 8), kListWarps * 32, lsmem, s>>>(
        j.f_packed.as<uint32_t>(), j.f_stride, t, perm, n, k, words, 32 - slots_log2, j.f_distinct.as<uint16_t>(),
        j.f_dstride, j.f_meta.as<int4>(), j.f_repeats.as<uint32_t>(), j.f_hist.as<uint32_t>() + K4, ctl, most);
    count_launch(ctx);
    CRISPY_CK(ctx, cudaGetLastError());
    return CRISPY_OK;
}
}  // namespace

// One pass over the pairs whose lower read ID lies in [olo, ohi): survivors
// in j.keys / j.vals (up to cap), their count in j.counter (cleared by the
// caller) and *total.  *gave_up: the candidates are more than their buffer
// takes; the caller then runs the tile kernels instead.  The threshold tables must
// be in j.mmin / j.smin.
int kmer_filter_pass(crispy_ctx* ctx, int olo, int ohi, int64_t cap, int A, int sd, int64_t* total,
                     bool* gave_up) {
    KmerJob& j = ctx->kmer;
    cudaStream_t s = ctx->stream;
    const int n = j.n, k = j.k;
    const int panels = (n + kRows - 1) / kRows;
    const int tiles = (n + kCols - 1) / kCols;
    *gave_up = false;
    *total = 0;
    CRISPY_TRY(ensure(ctx, j.f_need, (size_t)n * 4));
    CRISPY_TRY(ensure(ctx, j.f_cmin, (size_t)((n + 31) / 32) * 4));
    CRISPY_TRY(ensure(ctx, j.f_ctl, sizeof(FilterCtl)));
    if (k == 8) {
        CRISPY_TRY(ensure(ctx, j.f_heavy, (size_t)n));
        CRISPY_TRY(ensure(ctx, j.f_pend, (size_t)panels * 4));
    }
    FilterCtl* ctl = j.f_ctl.as<FilterCtl>();
    const int32_t* t = k == 8 ? j.f_t.as<int32_t>() : j.t0.as<int32_t>();
    CRISPY_CK(ctx, cudaMemsetAsync(ctl, 0, sizeof(FilterCtl), s));
    filter_need_kernel<<<(n + 255) / 256, 256, 0, s>>>(t, j.smin.as<uint16_t>(), j.mmin.as<uint16_t>(),
                                                       k == 8 ? j.f_nh.as<uint16_t>() : nullptr, n,
                                                       j.f_need.as<float>(), j.f_cmin.as<float>(),
                                                       k == 8 ? j.f_heavy.as<uint8_t>() : nullptr, ctl);
    count_launch(ctx);
    // columns of each panel: from its own rows to the last read (K = 8: to
    // the end of its last row's H key, unless a read is H-heavy)
    pinned_vector<int32_t>& pend = j.h_pend;
    if (k == 8) {
        filter_panel_end_kernel<<<(panels + 127) / 128, 128, 0, s>>>(j.f_hkey.as<uint32_t>(), n, panels,
                                                                     j.f_pend.as<int32_t>());
        count_launch(ctx);
        pend.resize(panels + 1);
        CRISPY_CK(ctx, cudaMemcpyAsync(pend.data(), j.f_pend.ptr, (size_t)panels * 4, cudaMemcpyDeviceToHost, s));
        CRISPY_CK(ctx, cudaMemcpyAsync(pend.data() + panels, &ctl->any_heavy, 4, cudaMemcpyDeviceToHost, s));
        CRISPY_CK(ctx, cudaStreamSynchronize(s));
        if (pend[panels]) pend.clear();
    } else {
        pend.clear();
    }
    const int plo = k == 8 ? 0 : olo / kRows, phi = k == 8 ? panels : (ohi + kRows - 1) / kRows;
    int64_t work = 0;
    auto first_tile = [&](int p) { return kRows * p / kCols; };
    auto end_tile = [&](int p) { return pend.empty() ? tiles : (pend[p] + kCols - 1) / kCols; };
    for (int p = plo; p < phi; ++p) work += end_tile(p) - first_tile(p);
    // rounds of at most 2^33 pairs; segments: four per block and round, at
    // least one tile each
    const int64_t pairs = work * kRows * kCols;
    const int rounds = (int)std::min<int64_t>(kMaxRounds, std::max<int64_t>(1, (pairs + (1ll << 33) - 1) >> 33));
    const int64_t nsegs = std::max<int64_t>(1, std::min<int64_t>(work, 4ll * ctx->sm_count * rounds));
    std::vector<int4>& items = j.h_items;
    std::vector<int2>& segs = j.h_segs;   // the probe's, then the rounds'
    items.clear();
    segs.clear();
    const int64_t room = candidate_room((pairs + rounds - 1) / rounds, k), ccap = candidate_buffer(room);
    const bool probe = work >= kProbeFrom * ctx->sm_count && room * rounds < (int64_t)n * (n - 1) / 2;
    const int64_t nprobe = probe ? ctx->sm_count : 0;
    const int64_t probe_run = std::min<int64_t>(8, std::max<int64_t>(1, work / (128ll * ctx->sm_count)));
    segs.resize(nprobe);
    int64_t done = 0, probed = 0, probe_tiles = 0;
    bool open = false;   // the open segment's first tiles go to the probe
    for (int p = plo; p < phi; ++p) {
        for (int a = first_tile(p), e = end_tile(p); a < e;) {
            const int64_t seg = (int64_t)segs.size() - nprobe;
            if (done == work * seg / nsegs) {
                if (seg > 0) segs.back().y = (int)items.size();
                segs.push_back(make_int2((int)items.size(), 0));
                open = probed < nprobe && probed < (seg + 1) * nprobe / nsegs;
                continue;
            }
            const int64_t left = work * seg / nsegs - done;   // tiles to the end of the open segment
            int c = (int)std::min<int64_t>(e - a, left);
            if (open) {
                c = (int)std::min<int64_t>(c, probe_run);
                segs[probed++] = make_int2((int)items.size(), (int)items.size() + 1);
                segs.back().x = (int)items.size() + 1;
                probe_tiles += c;
                open = false;
            }
            items.push_back(make_int4(p, a, a + c, 0));
            a += c;
            done += c;
        }
    }
    if (items.empty()) return CRISPY_OK;
    segs.back().y = (int)items.size();
    const size_t item_bytes = items.size() * sizeof(int4);
    CRISPY_TRY(ensure(ctx, j.f_items, item_bytes + segs.size() * sizeof(int2)));
    CRISPY_CK(ctx, cudaMemcpyAsync(j.f_items.ptr, items.data(), item_bytes, cudaMemcpyHostToDevice, s));
    CRISPY_CK(ctx, cudaMemcpyAsync(j.f_items.as<char>() + item_bytes, segs.data(), segs.size() * sizeof(int2),
                                   cudaMemcpyHostToDevice, s));
    CRISPY_TRY(ensure(ctx, j.f_cand, (size_t)ccap * sizeof(uint2)));
    CRISPY_TRY(ensure(ctx, j.f_candidx, (size_t)ccap * 4));
    CRISPY_TRY(ensure(ctx, j.f_sorted, (size_t)ccap * sizeof(uint2)));
    CRISPY_TRY(ensure(ctx, j.f_rows, (size_t)n * 8));
    CRISPY_CK(ctx, cudaMemsetAsync(j.f_rows.ptr, 0, (size_t)n * 4, s));

    const int chunks = j.f_dims / 256;
    const bool resident = chunks <= kResidentChunks;
    const size_t fixed = 1024 + kEpilogueWarps * kCandBuf * sizeof(uint2) + sizeof(Bars);
    const size_t bytes_a = resident ? (size_t)chunks * kChunkA : 0;
    const size_t stage = resident ? kChunkB : kChunkA + kChunkB;
    const int depth = (int)std::min<size_t>(kMaxDepth, (kSmemLimit - fixed - bytes_a) / (2 * stage));
    const size_t smem = fixed + bytes_a + 2 * depth * stage;
    auto kern = resident ? kmer_filter_kernel<true> : kmer_filter_kernel<false>;
    CRISPY_TRY(open_smem(ctx, kern));
    CUtensorMap map_rows, map_cols;
    CRISPY_TRY(signature_map(ctx, &map_rows, j.f_sig.ptr, j.f_dims / 2, n, kRows));
    CRISPY_TRY(signature_map(ctx, &map_cols, j.f_sig.ptr, j.f_dims / 2, n, kCols));

    FilterArgs fa{};
    fa.chunks = chunks;
    fa.depth = depth;
    fa.n = n;
    fa.need = j.f_need.as<float>();
    fa.cmin = j.f_cmin.as<float>();
    fa.excess = j.f_excess.as<uint16_t>();
    fa.cand = j.f_cand.as<uint2>();
    fa.cap = (unsigned long long)ccap;
    fa.ctl = ctl;
    fa.wait = kWaitCycles;
    if (const char* e = std::getenv("CRISPY_KMER_WAIT")) fa.wait = std::atoll(e);
    VerifyArgs va{};
    va.cand = fa.cand;
    va.cap = fa.cap;
    va.ctl = ctl;
    va.sorted = j.f_sorted.as<uint2>();
    va.candidx = j.f_candidx.as<uint32_t>();
    va.rowcnt = j.f_rows.as<uint32_t>();
    va.rowoff = va.rowcnt + n;
    va.distinct = j.f_distinct.as<uint16_t>();
    va.dstride = j.f_dstride;
    va.meta = j.f_meta.as<int4>();
    va.repeats = j.f_repeats.as<uint32_t>();
    va.perm = k == 8 ? j.f_perm.as<int32_t>() : nullptr;
    va.hkey = k == 8 ? j.f_hkey.as<uint32_t>() : nullptr;
    va.heavy = k == 8 ? j.f_heavy.as<uint8_t>() : nullptr;
    va.mmin = j.mmin.as<uint16_t>();
    va.n = n;
    va.K = k;
    va.rep_slots = rep_slots_for(k, j.max_t);
    va.repeated = j.f_hist.as<uint32_t>() + (1 << (2 * k));
    va.tuples = (float)std::max<int64_t>(j.sum_t, 1);
    va.most = (double)candidates_worth((pairs + rounds - 1) / rounds, k);
    va.olo = olo;
    va.ohi = ohi;
    va.A = A;
    va.sd = sd;
    va.counter = j.counter.as<unsigned long long>();
    va.keys = j.keys.as<uint64_t>();
    va.vals = j.vals.as<uint32_t>();
    va.out_cap = cap;
    // byte marks where they leave room for five blocks per SM
    const bool bytes = k <= 6 && (size_t)kVerifyWarps * ((1 << (2 * k)) + va.rep_slots * 4) <= kSmemLimit / 5;
    const int map_words = bytes ? 1 << (2 * k - 2) : 1 << (2 * k - 5);
    const size_t vsmem = (size_t)kVerifyWarps * (map_words + va.rep_slots) * 4;
    auto verify = bytes ? filter_verify_kernel<true, false>
                        : k < 8 ? filter_verify_kernel<false, false> : filter_verify_kernel<false, true>;
    CRISPY_TRY(open_smem(ctx, verify));
    int per_sm = 1;
    cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, verify, kVerifyWarps * 32, vsmem);
    per_sm = std::max(1, per_sm);
    ev_begin(ctx, ctx->ev_kmer, s);
    fa.items = j.f_items.as<int4>();
    const int cgrid = std::min((n + 63) / 64, ctx->sm_count * 8);
    const int2* d_segs = reinterpret_cast<const int2*>(j.f_items.as<char>() + item_bytes);
    if (probe) {
        fa.segs = d_segs;
        fa.nsegs = (int)nprobe;
        fa.round = 0;
        kern<<<(unsigned)nprobe, kFilterThreads, smem, s>>>(map_rows, map_cols, fa);
        count_launch(ctx);
    }
    const unsigned long long most = probe ? (unsigned long long)((double)room * rounds * probe_tiles / work) : ~0ull;
    if (!j.f_lists) {
        CRISPY_TRY(build_lists(ctx, ctl, most));
    } else if (probe) {
        filter_probe_kernel<<<1, 1, 0, s>>>(ctl, most);
        count_launch(ctx);
    }
    for (int r = 0; r < rounds; ++r) {
        const int64_t i0 = nsegs * r / rounds, i1 = nsegs * (r + 1) / rounds;
        if (i1 <= i0) continue;
        fa.segs = d_segs + nprobe + i0;
        fa.nsegs = (int)(i1 - i0);
        fa.round = va.round = r;
        kern<<<(unsigned)std::min<int64_t>(ctx->sm_count, i1 - i0), kFilterThreads, smem, s>>>(map_rows, map_cols, fa);
        filter_count_kernel<<<cgrid, 256, 0, s>>>(va);
        filter_rows_kernel<<<(n + 255) / 256, 256, 0, s>>>(va);
        filter_scatter_kernel<<<cgrid, 256, 0, s>>>(va);
        verify<<<ctx->sm_count * per_sm, kVerifyWarps * 32, vsmem, s>>>(va);
        count_launch(ctx, 5);
    }
    ev_end(ctx, ctx->ev_kmer, s);
    ctx->stats.kmer_launches += rounds;
    CRISPY_CK(ctx, cudaGetLastError());
    FilterCtl h;
    unsigned long long found = 0;
    CRISPY_CK(ctx, cudaMemcpyAsync(&h, ctl, sizeof(h), cudaMemcpyDeviceToHost, s));
    CRISPY_CK(ctx, cudaMemcpyAsync(&found, j.counter.ptr, sizeof(found), cudaMemcpyDeviceToHost, s));
    CRISPY_CK(ctx, cudaStreamSynchronize(s));
    *total = (int64_t)found;
    if (h.timeout) return fail(ctx, CRISPY_E_TIMEOUT, "k-mer filter: a device-side wait ran out");
    *gave_up = h.overflow != 0;
    if (!*gave_up) j.f_lists = true;
    int64_t cand = 0;
    for (int r = 0; r < rounds; ++r) cand += (int64_t)h.cand[r];
    j.f_pairs += pairs;
    j.f_found += cand;
    return CRISPY_OK;
}

}  // namespace crispy
