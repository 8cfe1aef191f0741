// pre.cu -- preprocess on GB300: read filters and duplicate merge.
//
// The reference (preprocess.cpp) keeps its reads in a std::list and, after
// the optional filters, sorts the whole list by (length, strcmp) with the
// list's stable merge sort and folds each run of equal sequences into its
// last read (mergeReads, :244-280).  Here the records go to the device once
// and everything after the host-side length statistics runs there:
//   1. pre_pad_kernel copies every read to a 16-byte aligned slot (zero
//      padded), so byte-wise comparisons become 128-bit loads;
//   2. pre_filter_kernel applies the length cut and the N/n check of
//      processReadLength (:322-392);
//   3. pre_primer_kernel runs SWLocalAlignment (:394-527) of the primer
//      against each read's first 2 x primer-length bytes, one thread per
//      read with its DP rows in shared memory;
//   4. the surviving read indices are sorted by (length, bytes, record
//      index): 1024-index tiles by a bitonic network in shared memory, then
//      merge passes in which each index finds its place in the partner run
//      by binary search, both on 128-bit keys (pre_key_kernel) that stand for
//      the length and the first 28 bytes.  The record index as last key makes every key
//      distinct, so the order equals the reference's stable sort;
//   5. pre_last_kernel flags the last read of each run of equal sequences;
//      compaction of those flags gives the kept reads and, from the gaps
//      between them, each run's size (the merged frequency: every read that
//      reaches the merge has frequency 1).
// Comparisons read the reads from L2: the padded copy of 100,000 reads of
// 300-500 bases is about 42 MB.
#include <cuda_runtime.h>

#include <algorithm>
#include <climits>
#include <cmath>
#include <cstring>
#include <vector>

#include "internal.h"

namespace crispy {
namespace {

constexpr uint32_t kNone = 0xffffffffu;   // tile padding: sorts after every read
constexpr int kTile = 1024;               // indices per bitonic tile
constexpr int kTileThreads = kTile / 2;
constexpr int kMaxPrimer = 256;           // primer bases the shared-memory DP rows allow

struct ReadSet {
    const uint4* pad;      // reads, each at a 16-byte aligned slot, zero padded
    const int64_t* woff;   // first 16-byte word of each read
    const int32_t* len;
};

__device__ __forceinline__ uint32_t be32(uint32_t x) { return __byte_perm(x, 0, 0x0123); }

// strcmp-style order of two reads of equal length L (unsigned bytes) whose
// first `first` 16-byte words are equal.
__device__ __forceinline__ int cmp_bytes(const ReadSet& r, uint32_t a, uint32_t b, int L, int first = 0) {
    const uint4* pa = r.pad + r.woff[a];
    const uint4* pb = r.pad + r.woff[b];
    const int nw = (L + 15) >> 4;
    // four words of each on their way at a time: duplicates compare to the end
    for (int w0 = first; w0 < nw; w0 += 4) {
        uint4 xs[4], ys[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int w = min(w0 + q, nw - 1);
            xs[q] = __ldg(pa + w);
            ys[q] = __ldg(pb + w);
        }
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const uint4 x = xs[q], y = ys[q];
            if (x.x != y.x) return be32(x.x) < be32(y.x) ? -1 : 1;
            if (x.y != y.y) return be32(x.y) < be32(y.y) ? -1 : 1;
            if (x.z != y.z) return be32(x.z) < be32(y.z) ? -1 : 1;
            if (x.w != y.w) return be32(x.w) < be32(y.w) ? -1 : 1;
        }
    }
    return 0;
}

// READ::operator< (preprocess.cpp:42-49) with the record index as last key.
__device__ __forceinline__ bool read_less(const ReadSet& r, uint32_t a, uint32_t b) {
    if (b == kNone) return a != kNone;
    if (a == kNone) return false;
    const int la = __ldg(r.len + a), lb = __ldg(r.len + b);
    if (la != lb) return la < lb;
    const int c = cmp_bytes(r, a, b, la);
    return c ? c < 0 : a < b;
}

// Sort key of a read: its length (16 bits, saturated) and its first 28 bytes
// as 4-bit classes that keep their order -- one class for each of NUL, A, C,
// G, N and T, one for every range between them.  A byte of a range ends the
// key (zeros follow; a length that does not fit leaves no class at all), so
// two reads whose keys differ are in the order of their keys, and two whose
// keys agree need the full comparison.
struct ReadKey {
    unsigned long long hi, lo;
};
__device__ __forceinline__ bool key_equal(const ReadKey& a, const ReadKey& b) { return a.hi == b.hi && a.lo == b.lo; }
// Order of two reads of this key: their length is known, and where no range
// is among the first 16 classes (odd ones) so are their first 16 bytes.
__device__ __forceinline__ int tie_cmp(const ReadSet& r, const ReadKey& k, uint32_t a, uint32_t b) {
    const int L = (int)(k.hi >> 48);
    const bool exact = (k.hi & 0x0000111111111111ull) == 0 && (k.lo & 0x1111000000000000ull) == 0;
    return cmp_bytes(r, a, b, L, exact ? 1 : 0);
}
// kWhole: reads whose keys agree are compared; otherwise they keep the record
// order, to be settled group by group afterwards.
template <bool kWhole>
__device__ __forceinline__ bool key_less(const ReadSet& r, const ReadKey& ka, uint32_t a, const ReadKey& kb, uint32_t b) {
    if (ka.hi != kb.hi) return ka.hi < kb.hi;
    if (ka.lo != kb.lo) return ka.lo < kb.lo;
    if (!kWhole) return a < b;
    if (a == kNone || b == kNone || (ka.hi >> 48) == 0xFFFFull) return read_less(r, a, b);
    const int c = tie_cmp(r, ka, a, b);
    return c ? c < 0 : a < b;
}
__device__ __forceinline__ uint32_t byte_class(uint32_t c) {
    if (c == 0) return 0;
    if (c < 'A') return 1;
    if (c == 'A') return 2;
    if (c < 'C') return 3;
    if (c == 'C') return 4;
    if (c < 'G') return 5;
    if (c == 'G') return 6;
    if (c < 'N') return 7;
    if (c == 'N') return 8;
    if (c < 'T') return 9;
    return c == 'T' ? 10 : 11;
}
__global__ void pre_key_kernel(ReadSet r, const uint32_t* __restrict__ idx, int64_t m, ReadKey* __restrict__ keys) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const uint32_t x = idx[i];
    const int L = r.len[x];
    const uint4* p = r.pad + r.woff[x];
    const uint4 zero = make_uint4(0u, 0u, 0u, 0u);
    const uint4 w0 = L > 0 ? __ldg(p) : zero, w1 = L > 16 ? __ldg(p + 1) : zero;
    const uint32_t words[7] = {w0.x, w0.y, w0.z, w0.w, w1.x, w1.y, w1.z};
    unsigned long long hi = (unsigned long long)min(L, 0xFFFF) << 48, lo = 0;
    bool open = L < 0xFFFF;
#pragma unroll
    for (int q = 0; q < 28; ++q) {
        const uint32_t c = open ? byte_class((words[q / 4] >> (8 * (q % 4))) & 0xFFu) : 0u;
        if (q < 12) hi |= (unsigned long long)c << (44 - 4 * q);
        else lo |= (unsigned long long)c << (60 - 4 * (q - 12));
        open = open && (c & 1u) == 0u;
    }
    keys[i] = ReadKey{hi, lo};
}

__global__ void pre_pad_kernel(const uint8_t* __restrict__ seq, const int64_t* __restrict__ off,
                               const int32_t* __restrict__ len, const int64_t* __restrict__ woff,
                               int n, uint4* __restrict__ pad) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t r = warp; r < n; r += nwarps) {
        const uint8_t* src = seq + off[r];
        const int L = len[r];
        uint4* dst = pad + woff[r];
        for (int w = lane; w < (L + 15) >> 4; w += 32) {
            uint32_t v[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                uint32_t word = 0;
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const int p = 16 * w + 4 * q + b;
                    word |= (uint32_t)(p < L ? src[p] : 0u) << (8 * b);
                }
                v[q] = word;
            }
            dst[w] = make_uint4(v[0], v[1], v[2], v[3]);
        }
    }
}

// alive = frequency != 0, then (with the length check) the length cut and
// the N/n test of processReadLength.  counters[0]: reads cut by length,
// counters[1]: reads dropped for N/n.
__global__ void pre_filter_kernel(ReadSet r, const uint8_t* __restrict__ freq, int n, int length_check,
                                  unsigned long long lo, unsigned long long hi,
                                  uint8_t* __restrict__ alive, unsigned int* __restrict__ counters) {
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t i = warp; i < n; i += nwarps) {
        bool a = freq[i] != 0;
        if (a && length_check) {
            const int L = r.len[i];
            const unsigned long long ul = (unsigned long long)L;
            if (ul < lo || ul > hi) {
                a = false;
                if (lane == 0) atomicAdd(&counters[0], 1u);
            } else {
                const uint4* p = r.pad + r.woff[i];
                bool hit = false;
                for (int w = lane; w < (L + 15) >> 4 && !hit; w += 32) {
                    const uint4 x = p[w];
                    // a byte is N or n iff (byte | 0x20) == 'n'; padding bytes are 0
                    hit = __vcmpeq4(x.x | 0x20202020u, 0x6e6e6e6eu) | __vcmpeq4(x.y | 0x20202020u, 0x6e6e6e6eu) |
                          __vcmpeq4(x.z | 0x20202020u, 0x6e6e6e6eu) | __vcmpeq4(x.w | 0x20202020u, 0x6e6e6e6eu);
                }
                if (__any_sync(0xffffffffu, hit)) {
                    a = false;
                    if (lane == 0) atomicAdd(&counters[1], 1u);
                }
            }
        }
        if (lane == 0) alive[i] = a ? 1 : 0;
    }
}

// SWLocalAlignment (preprocess.cpp:394-527) of the primer A (m bases)
// against B = the first min(2m, L) bytes of each alive read, and the
// decision of processPrimer (:530-560): the read goes when the best local
// alignment's start equals its end.  Scores: match +4, mismatch -1, gap -2,
// floor 0; ties of a cell go to 0, then diagonal, then the cell above (row
// i-1), then the left one; the best cell is the first in row-major order
// with the highest score and, among those, the fewest mismatches.  One
// thread per read; the previous row (score, start, mismatches) lives in
// shared memory as int16, laid out [column][thread].  counters[2] counts the
// reads dropped.
__global__ void pre_primer_kernel(ReadSet r, int n, const uint8_t* __restrict__ primer, int m, int max_mm,
                                  uint8_t* __restrict__ alive, unsigned int* __restrict__ counters) {
    extern __shared__ int16_t rows[];
    const int T = blockDim.x, t = threadIdx.x;
    const int cols = 2 * m + 1;
    int16_t* S = rows;
    int16_t* ST = rows + cols * T;
    int16_t* MM = rows + 2 * cols * T;
    const int64_t stride = (int64_t)gridDim.x * T;
    for (int64_t i0 = (int64_t)blockIdx.x * T + t; i0 < n; i0 += stride) {
        if (!alive[i0]) continue;
        const int L = r.len[i0];
        const int lb = min(2 * m, L);
        const uint8_t* B = reinterpret_cast<const uint8_t*>(r.pad + r.woff[i0]);
        for (int j = 0; j <= lb; ++j) { S[j * T + t] = 0; ST[j * T + t] = 0; MM[j * T + t] = 0; }
        int best = -9999, best_mm = 999, startA = 0, endA = 0;
        for (int i = 1; i <= m; ++i) {
            const uint8_t a = primer[i - 1];
            int dS = S[t], dST = ST[t], dMM = MM[t];   // row i-1, column 0
            int lS = 0, lST = i, lMM = 0;               // row i, column 0
            S[t] = 0; ST[t] = (int16_t)i; MM[t] = 0;
            for (int j = 1; j <= lb; ++j) {
                const int uS = S[j * T + t], uST = ST[j * T + t], uMM = MM[j * T + t];
                const bool eq = a == B[j - 1];
                const int t0 = dS + (eq ? 4 : -1), t1 = uS - 2, t2 = lS - 2;
                const int s = max(max(max(t0, t1), t2), 0);
                int st, mm;
                if (s == 0) { st = i - 1; mm = 0; }
                else if (s == t0) { st = dST; mm = dMM + (eq ? 0 : 1); }
                else if (s == t1) { st = uST; mm = uMM + 1; }
                else { st = lST; mm = lMM + 1; }
                if (best < s || (best == s && best_mm > mm)) { best = s; startA = st; endA = i; best_mm = mm; }
                S[j * T + t] = (int16_t)s; ST[j * T + t] = (int16_t)st; MM[j * T + t] = (int16_t)mm;
                dS = uS; dST = uST; dMM = uMM;
                lS = s; lST = st; lMM = mm;
            }
        }
        const int total = best_mm + startA + abs(m - endA);
        const int s0 = total <= max_mm ? startA : 0, e0 = total <= max_mm ? endA : 0;
        if (s0 == e0) {
            alive[i0] = 0;
            atomicAdd(&counters[2], 1u);
        }
    }
}

// Comparisons inside groups of equal keys up to which settling them costs less
// than comparing reads in every merge: 4 million, whatever the number of reads
// (20,000 reads of 250 nt settled with 2.5 M in 430 us and compared throughout
// in 499, with 4.5 M 539 and 513; 60,000 with 3.3 M 622 and 632, with 18 M 864
// and 658; 150,000 with 4.9 M 1,026 and 983, of 120 nt with 6.2 M 930 and 808).
// An estimate that was wrong by more than four times is given up for the other
// form.
constexpr double kSettleWorth = 4e6;
constexpr unsigned long long kSettleMost = 1ull << 24;

// Whether reads of equal keys are so many that comparing the reads throughout
// costs less than settling them group by group.  force: the reads are compared
// throughout, whatever the estimate says.
struct Ties {
    const unsigned long long* too_many;   // pre_sample_kernel
    bool force;
    __device__ bool many() const { return force || *too_many != 0; }
};

// The estimate: pairs of equal keys among up to 1,024 reads spread over the
// set (found in a table of hashes), and as many more in the whole set as it
// has more pairs.  One block, before the sort (5 us): looking at sorted tiles
// instead costs sets with many ties a tile sort more (28 us).  Whole calls of
// 60,000 reads of 250 nt, reads compared throughout without keys, and now: no
// common head 642 and 556 us, a common head of 20 bases 695 and 652, of 40
// bases 714 and 674, all of one length 739 and 650.
constexpr int kSample = 1024, kSampleSlots = 2048;
static_assert(kSampleSlots >= 2 * kSample && kSampleSlots * 12 + 16 <= 48 * 1024, "a free slot for every read, in static shared memory");
__global__ void __launch_bounds__(kSample) pre_sample_kernel(const ReadKey* __restrict__ keys, int64_t m, double limit,
                                                             unsigned long long* __restrict__ too_many) {
    __shared__ unsigned long long slot[kSampleSlots];
    __shared__ unsigned count[kSampleSlots];
    __shared__ unsigned pairs;
    const int t = threadIdx.x;
    for (int q = t; q < kSampleSlots; q += kSample) { slot[q] = 0; count[q] = 0; }
    if (t == 0) pairs = 0;
    __syncthreads();
    const int64_t step = m / kSample;   // 0: every read
    if (step > 0 || t < m) {
        const int64_t p = step > 0 ? t * step + (int64_t)((uint32_t)t * 0x9E3779B1u >> 8) % step : t;
        const ReadKey k = keys[p];
        const unsigned long long h = ((k.hi ^ (k.lo << 1 | k.lo >> 63)) * 0x9E3779B97F4A7C15ull ^ k.lo * 0xC2B2AE3D27D4EB4Full) | 1ull;
        for (unsigned q = (unsigned)(h >> 40) % kSampleSlots;; q = (q + 1) % kSampleSlots) {
            const unsigned long long old = atomicCAS(&slot[q], 0ull, h);
            if (old == 0 || old == h) {
                const unsigned before = atomicAdd(&count[q], 1u);
                if (before) atomicAdd(&pairs, before);
                break;
            }
        }
    }
    __syncthreads();
    const double more = step > 0 ? (double)m / kSample : 1.0;
    if (t == 0) *too_many = 2.0 * pairs * more * more > limit ? 1ull : 0ull;
}

// Bitonic sort of one tile: keys and indices in shared memory.  With kWhole
// the reads themselves are looked at where keys agree; a single such pair
// makes its whole block wait for loads that depend on one another (85 us for
// 60,000 reads, 152 with all reads compared at every step).
template <bool kWhole>
__global__ void __launch_bounds__(kTileThreads) pre_tile_sort_kernel(uint32_t* idx, ReadKey* keys, int64_t m,
                                                                     ReadSet r, const Ties ties) {
    if (kWhole != ties.many()) return;
    __shared__ uint32_t s[kTile];
    __shared__ ReadKey sk[kTile];
    const int64_t base = (int64_t)blockIdx.x * kTile;
    for (int t = threadIdx.x; t < kTile; t += kTileThreads) {
        s[t] = base + t < m ? idx[base + t] : kNone;
        sk[t] = base + t < m ? keys[base + t] : ReadKey{~0ull, ~0ull};
    }
    __syncthreads();
    for (int k = 2; k <= kTile; k <<= 1) {
        for (int j = k >> 1; j > 0; j >>= 1) {
            const int t = threadIdx.x;
            const int i = 2 * t - (t & (j - 1));   // bit j of i is clear; partner i + j
            const uint32_t a = s[i], b = s[i + j];
            const ReadKey ka = sk[i], kb = sk[i + j];
            const bool up = (i & k) == 0;
            if (up ? key_less<kWhole>(r, kb, b, ka, a) : key_less<kWhole>(r, ka, a, kb, b)) {
                s[i] = b; s[i + j] = a;
                sk[i] = kb; sk[i + j] = ka;
            }
            __syncthreads();
        }
    }
    for (int t = threadIdx.x; t < kTile; t += kTileThreads)
        if (base + t < m) {
            idx[base + t] = s[t];
            keys[base + t] = sk[t];
        }
}

// One merge pass over sorted runs of `width`: each index moves to its
// position in the merged pair of runs, found by a binary search for the
// number of smaller reads in the partner run (one load of a key per step
// unless the reads have to be compared).
__global__ void pre_merge_kernel(const uint32_t* __restrict__ src, const ReadKey* __restrict__ skey,
                                 uint32_t* __restrict__ dst, ReadKey* __restrict__ dkey, int64_t m,
                                 int64_t width, ReadSet r, const Ties ties) {
    const bool whole = ties.many();
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= m) return;
    const int64_t run = i / width;
    const int64_t base = (run & ~1LL) * width;
    const uint32_t x = src[i];
    const ReadKey kx = skey[i];
    int64_t lo, hi, p0, pos;
    if ((run & 1) == 0) {
        p0 = base + width;
        if (p0 >= m) { dst[i] = x; dkey[i] = kx; return; }
        lo = p0; hi = min(base + 2 * width, m);
        pos = i - base;
    } else {
        p0 = base;
        lo = base; hi = base + width;
        pos = i - (base + width);
    }
    while (lo < hi) {
        const int64_t mid = (lo + hi) >> 1;
        const ReadKey km = skey[mid];
        const uint32_t xm = src[mid];
        if (whole ? key_less<true>(r, km, xm, kx, x) : key_less<false>(r, km, xm, kx, x)) lo = mid + 1;
        else hi = mid;
    }
    const int64_t to = base + pos + (lo - p0);
    dst[to] = x;
    dkey[to] = kx;
}

// Groups of equal keys.  One warp per position finds its group's range; the
// group's first position adds its comparisons to *work.
constexpr unsigned kGroupMost = 4096;   // larger groups count as too much work
constexpr unsigned long long kTooMuch = 1ull << 62;   // (the others' squares sum to 2^43 at the most)
__global__ void pre_group_kernel(const ReadKey* __restrict__ keys, int64_t m, uint2* __restrict__ range,
                                 unsigned long long* __restrict__ work, const Ties ties) {
    if (ties.many()) return;
    const unsigned full = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (p >= m) return;
    const ReadKey k = keys[p];
    int64_t lo = p, hi = p + 1;
    for (int run = 32; run == 32 && p - lo < kGroupMost;) {
        const int64_t q = lo - 1 - lane;
        const unsigned ne = ~__ballot_sync(full, q >= 0 && key_equal(keys[q], k));
        run = ne ? __ffs(ne) - 1 : 32;
        lo -= run;
    }
    for (int run = 32; run == 32 && hi - p <= kGroupMost;) {
        const int64_t q = hi + lane;
        const unsigned ne = ~__ballot_sync(full, q < m && key_equal(keys[q], k));
        run = ne ? __ffs(ne) - 1 : 32;
        hi += run;
    }
    if (lane == 0) {
        range[p] = make_uint2((uint32_t)lo, (uint32_t)hi);
        const unsigned long long g = (unsigned long long)(hi - lo);
        if (g >= kGroupMost) atomicOr(work, kTooMuch);
        else if (lo == p && g > 1) atomicAdd(work, g * g);
    }
}

// Each read's place in its group: one warp counts the group's reads that come
// before it.  Where the estimate missed groups so large that the merges are the
// better way after all (*work is above the limit) the groups stay unsettled,
// and dst is the order as it stands: the kernels that follow read it before
// the host learns that it has to sort again.
__global__ void pre_rank_kernel(const uint32_t* __restrict__ src, const uint2* __restrict__ range, int64_t m, ReadSet r,
                                const unsigned long long* __restrict__ work, unsigned long long limit,
                                uint32_t* __restrict__ dst, const Ties ties) {
    if (ties.many() || *work > limit) {          // sorted already, or not to be settled here
        const int64_t q = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
        if (q < m) dst[q] = src[q];
        return;
    }
    const int lane = threadIdx.x & 31;
    const int64_t p = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    if (p >= m) return;
    const uint32_t x = src[p];
    const uint2 g = range[p];
    unsigned before = 0;
    if (g.y - g.x > 1)
        for (uint32_t q = g.x + lane; q < g.y; q += 32) before += q != (uint32_t)p && read_less(r, src[q], x);
    before = __reduce_add_sync(0xffffffffu, before);
    if (lane == 0) dst[g.x + before] = x;
}

// flag[p] = 1 where sorted[p] is the last read of its run of equal sequences.
__global__ void pre_last_kernel(const uint32_t* __restrict__ sorted, const ReadKey* __restrict__ keys, int64_t m,
                                ReadSet r, uint8_t* __restrict__ flag) {
    const int64_t p = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= m) return;
    bool last = true;
    if (p + 1 < m && key_equal(keys[p], keys[p + 1])) {
        const uint32_t a = sorted[p], b = sorted[p + 1];
        const int la = r.len[a];
        last = la != r.len[b] || (la < 0xFFFF ? tie_cmp(r, keys[p], a, b) : cmp_bytes(r, a, b, la)) != 0;
    }
    flag[p] = last ? 1 : 0;
}

__global__ void pre_emit_kernel(const uint32_t* __restrict__ sorted, const uint32_t* __restrict__ pos,
                                int64_t kept, int32_t* __restrict__ out_idx, int32_t* __restrict__ out_freq) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kept) return;
    const int64_t p = pos[k];
    out_idx[k] = (int32_t)sorted[p];
    out_freq[k] = (int32_t)(p - (k ? (int64_t)pos[k - 1] : -1));
}

// Per kept read k (record out_idx[k]): its length as the stage's FASTA
// parser reads it back from the _Clean line "<seq>\n", its byte offset in
// the padded buffer, and bad[0] += 1 when the read holds a byte of
// deleteSpaces' set or is longer than 4,094 bytes.  For such reads that
// line does not come back as one piece with only the newline to trim.
// Otherwise the line loses the newline, then everything after its last
// base letter: ATGCatgc for kmerDist (kmerMain.cpp:289-295), nNATGCatgc for
// genDist (genMain.cpp:175-181); a read without one stays whole.
__global__ void pre_stage_kernel(ReadSet r, const int32_t* __restrict__ out_idx, int64_t kept, int flavour,
                                 int32_t* __restrict__ len_out, int64_t* __restrict__ off_out,
                                 unsigned int* __restrict__ bad) {
    const int64_t k = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (k >= kept) return;
    const int32_t i = out_idx[k];
    const int L = r.len[i];
    const uint8_t* b = reinterpret_cast<const uint8_t*>(r.pad + r.woff[i]);
    bool odd = L > 4094;
    int last = -1;
    for (int p = 0; p < L && !odd; ++p) {
        const uint8_t c = b[p];
        if ((c >= 8 && c <= 13) || c == ' ') odd = true;
        const uint8_t u = c & 0xDF;   // upper case
        if (u == 'A' || u == 'C' || u == 'G' || u == 'T' || (flavour && u == 'N')) last = p;
    }
    if (odd) atomicAdd(bad, 1u);
    len_out[k] = last >= 0 ? last + 1 : L;
    off_out[k] = r.woff[i] * 16;
}

int grid_for(int64_t items, int per_block, int cap) {
    return (int)std::max<int64_t>(1, std::min<int64_t>((items + per_block - 1) / per_block, cap));
}

// (int) of a double as x86 and Arm both give it for values inside int's
// range; outside it the conversion saturates.
int to_int_sat(double v) {
    if (!(v == v)) return 0;
    if (v >= 2147483647.0) return INT_MAX;
    if (v <= -2147483648.0) return INT_MIN;
    return (int)v;
}

}  // namespace

int pre_stage_reads(crispy_ctx* ctx, const crispy_raw* raw, int flavour, const uint8_t** d_bytes,
                    size_t* bytes, const int64_t** d_off, std::vector<int32_t>& h_len) {
    PreJob& j = ctx->pre;
    if (!j.ready) return fail(ctx, CRISPY_E_STATE, "no preprocess result on this context");
    if (!raw || raw_records(raw) != j.n)
        return fail(ctx, CRISPY_E_INPUT, "the raw records are not those of the last preprocess call");
    const int64_t kept = j.kept;
    // a header line longer than one 4,095-byte piece would come back with
    // its tail read as sequence
    for (int64_t k = 0; k < kept; ++k)
        if (raw_header_line(raw, j.h_idx[k]) + 1 > 4095)
            return fail(ctx, CRISPY_E_UNSUPPORTED,
                        "a kept read's header line exceeds 4095 bytes: read the _Clean file instead");
    h_len.resize((size_t)kept);
    *d_bytes = j.pad.as<uint8_t>();
    *bytes = j.pad.bytes;
    *d_off = nullptr;
    if (kept == 0) return CRISPY_OK;
    cudaSetDevice(ctx->device);
    cudaStream_t s = ctx->stream;
    CRISPY_TRY(ensure(ctx, j.stage_len, (size_t)kept * 4));
    CRISPY_TRY(ensure(ctx, j.stage_off, (size_t)kept * 8));
    CRISPY_CK(ctx, cudaMemsetAsync(j.counters.ptr, 0, 64, s));
    ReadSet rs{j.pad.as<uint4>(), j.woff.as<int64_t>(), j.len.as<int32_t>()};
    pre_stage_kernel<<<(unsigned)((kept + 255) / 256), 256, 0, s>>>(
        rs, j.out_idx.as<int32_t>(), kept, flavour, j.stage_len.as<int32_t>(), j.stage_off.as<int64_t>(),
        j.counters.as<unsigned int>() + 3);
    count_launch(ctx);
    CRISPY_CK(ctx, cudaGetLastError());
    unsigned int bad = 0;
    CRISPY_CK(ctx, cudaMemcpyAsync(h_len.data(), j.stage_len.ptr, (size_t)kept * 4, cudaMemcpyDeviceToHost, s));
    CRISPY_CK(ctx, cudaMemcpyAsync(&bad, j.counters.as<unsigned int>() + 3, 4, cudaMemcpyDeviceToHost, s));
    CRISPY_CK(ctx, cudaStreamSynchronize(s));
    if (bad)
        return fail(ctx, CRISPY_E_UNSUPPORTED,
                    "%u kept reads hold whitespace or exceed 4094 bytes: read the _Clean file instead", bad);
    *d_off = j.stage_off.as<int64_t>();
    return CRISPY_OK;
}

}  // namespace crispy

using namespace crispy;

extern "C" int crispy_preprocess(crispy_ctx* ctx, const char* seqbuf, const int64_t* offsets,
                                 const int32_t* lengths, const uint8_t* freq, int32_t n,
                                 const crispy_pre_opts* opts, int32_t* out_index, int32_t* out_freq,
                                 crispy_pre_stats* stats) {
    if (!ctx) return fail(nullptr, CRISPY_E_INPUT, "NULL context");
    if (n < 0 || (n > 0 && (!seqbuf || !offsets || !lengths || !freq || !out_index || !out_freq)))
        return fail(ctx, CRISPY_E_INPUT, "NULL argument");
    crispy_pre_stats st{};
    const crispy_pre_opts o = opts ? *opts : crispy_pre_opts{0, 1.0, nullptr, 2};
    const int m_primer = o.primer ? (int)std::strlen(o.primer) : 0;
    if (o.primer && m_primer > kMaxPrimer)
        return fail(ctx, CRISPY_E_UNSUPPORTED, "primer of %d bases: at most %d are supported", m_primer, kMaxPrimer);
    int64_t total_bytes = 0, words = 0;
    std::vector<int64_t> woff((size_t)n);
    for (int32_t i = 0; i < n; ++i) {
        if (lengths[i] < 0 || offsets[i] < 0) return fail(ctx, CRISPY_E_INPUT, "negative offset or length");
        total_bytes = std::max(total_bytes, offsets[i] + lengths[i]);
        woff[i] = words;
        words += (lengths[i] + 15) / 16;
    }

    // processReadLength's statistics, in record order and in double as the
    // reference sums them (preprocess.cpp:333-372).  Without a single read
    // the reference reports an error and applies neither the cut nor the N
    // check; st.length_reads = 0 then switches both off.
    unsigned long long lo = 0, hi = ~0ull;
    if (o.length_check) {
        double sum_len = 0.0, num = 0.0;
        for (int32_t i = 0; i < n; ++i)
            if (freq[i]) { sum_len += (double)lengths[i]; num += 1.0; }
        if (num >= 1.0) {
            const double ave = sum_len / num;
            double sum_diff = 0.0;
            int min_len = 65535, max_len = 0;
            for (int32_t i = 0; i < n; ++i) {
                if (!freq[i]) continue;
                const double diff = (double)(size_t)lengths[i] - ave;
                sum_diff += diff * diff;
                min_len = std::min(min_len, lengths[i]);
                max_len = std::max(max_len, lengths[i]);
            }
            sum_diff = sum_diff / num;
            const double sd = std::sqrt(sum_diff);
            st.length_reads = (int32_t)num;
            st.min_len0 = min_len;
            st.max_len0 = max_len;
            min_len = std::max(min_len, to_int_sat(ave - o.sd_allowed * sd));
            max_len = std::min(max_len, to_int_sat(ave + o.sd_allowed * sd));
            st.min_len = min_len;
            st.max_len = max_len;
            st.ave_len = ave;
            st.sd = sd;
            // length() < minLen and length() > maxLen compare as size_t
            lo = (unsigned long long)(long long)min_len;
            hi = (unsigned long long)(long long)max_len;
        }
    }
    if (n == 0) {
        ctx->pre.ready = true;
        ctx->pre.kept = 0;
        ctx->pre.n = 0;
        ctx->pre.h_idx.clear();
        if (stats) *stats = st;
        return CRISPY_OK;
    }

    cudaSetDevice(ctx->device);
    cudaStream_t s = ctx->stream;
    PreJob& j = ctx->pre;
    j.ready = false;
    CRISPY_TRY(ensure(ctx, j.seq, (size_t)total_bytes + 16));
    CRISPY_TRY(ensure(ctx, j.off, (size_t)n * 8));
    CRISPY_TRY(ensure(ctx, j.len, (size_t)n * 4));
    CRISPY_TRY(ensure(ctx, j.freq, (size_t)n));
    CRISPY_TRY(ensure(ctx, j.woff, (size_t)n * 8));
    CRISPY_TRY(ensure(ctx, j.pad, (size_t)(words + 1) * 16));
    CRISPY_TRY(ensure(ctx, j.alive, (size_t)n));
    CRISPY_TRY(ensure(ctx, j.idx, (size_t)n * 4));
    CRISPY_TRY(ensure(ctx, j.idx_alt, (size_t)n * 4));
    CRISPY_TRY(ensure(ctx, j.flags, (size_t)n));
    CRISPY_TRY(ensure(ctx, j.pos, (size_t)n * 4));
    CRISPY_TRY(ensure(ctx, j.tiles, ((size_t)n / kScanTile + 2) * 4));
    CRISPY_TRY(ensure(ctx, j.out_idx, (size_t)n * 4));
    CRISPY_TRY(ensure(ctx, j.out_freq, (size_t)n * 4));
    CRISPY_TRY(ensure(ctx, j.counters, 64));
    CRISPY_CK(ctx, cudaMemcpyAsync(j.seq.ptr, seqbuf, (size_t)total_bytes, cudaMemcpyHostToDevice, s));
    CRISPY_CK(ctx, cudaMemcpyAsync(j.off.ptr, offsets, (size_t)n * 8, cudaMemcpyHostToDevice, s));
    CRISPY_CK(ctx, cudaMemcpyAsync(j.len.ptr, lengths, (size_t)n * 4, cudaMemcpyHostToDevice, s));
    CRISPY_CK(ctx, cudaMemcpyAsync(j.freq.ptr, freq, (size_t)n, cudaMemcpyHostToDevice, s));
    CRISPY_CK(ctx, cudaMemcpyAsync(j.woff.ptr, woff.data(), (size_t)n * 8, cudaMemcpyHostToDevice, s));
    CRISPY_CK(ctx, cudaMemsetAsync(j.counters.ptr, 0, 64, s));

    ReadSet rs{j.pad.as<uint4>(), j.woff.as<int64_t>(), j.len.as<int32_t>()};
    const int warp_grid = 8 * ctx->sm_count;   // 256-thread blocks, 8 warps each
    pre_pad_kernel<<<grid_for((int64_t)n * 32, 256, warp_grid), 256, 0, s>>>(
        j.seq.as<uint8_t>(), j.off.as<int64_t>(), j.len.as<int32_t>(), j.woff.as<int64_t>(), n, j.pad.as<uint4>());
    pre_filter_kernel<<<grid_for((int64_t)n * 32, 256, warp_grid), 256, 0, s>>>(
        rs, j.freq.as<uint8_t>(), n, st.length_reads > 0 ? 1 : 0, lo, hi, j.alive.as<uint8_t>(),
        j.counters.as<unsigned int>());
    count_launch(ctx, 2);
    if (o.primer) {
        CRISPY_TRY(ensure(ctx, j.primer, (size_t)m_primer + 16));
        if (m_primer) CRISPY_CK(ctx, cudaMemcpyAsync(j.primer.ptr, o.primer, (size_t)m_primer, cudaMemcpyHostToDevice, s));
        const size_t per_thread = (size_t)3 * (2 * m_primer + 1) * sizeof(int16_t);
        int threads = (int)std::min<size_t>(256, (size_t)(96 * 1024) / per_thread);
        threads = std::max(32, threads / 32 * 32);
        const size_t smem = per_thread * threads;
        CRISPY_TRY(open_smem(ctx, pre_primer_kernel));
        pre_primer_kernel<<<grid_for(n, threads, 4 * ctx->sm_count), threads, smem, s>>>(
            rs, n, j.primer.as<uint8_t>(), m_primer, o.max_mismatches, j.alive.as<uint8_t>(),
            j.counters.as<unsigned int>());
        count_launch(ctx);
    }
    CRISPY_CK(ctx, cudaGetLastError());

    // alive records -> indices (record order)
    int64_t m = 0;
    CRISPY_TRY(compact_flags(ctx, s, j.alive.as<uint8_t>(), n, j.idx.as<uint32_t>(), j.tiles.as<uint32_t>(),
                             j.tmp, &m));
    unsigned int cnt[4] = {0, 0, 0, 0};
    CRISPY_CK(ctx, cudaMemcpyAsync(cnt, j.counters.ptr, sizeof cnt, cudaMemcpyDeviceToHost, s));

    // sort by (length, bytes, record index)
    uint32_t* a = j.idx.as<uint32_t>();
    uint32_t* b = j.idx_alt.as<uint32_t>();
    // keys and group ranges where the raw reads were (the padded ones stay),
    // as far as they reach: 40 bytes a read
    size_t carved = 0;
    auto carve = [&](DevBuf& own, size_t bytes, void** out) -> int {
        bytes = (std::max<size_t>(bytes, 1) + 255) / 256 * 256;
        if (carved + bytes <= j.seq.bytes) {
            *out = j.seq.as<uint8_t>() + carved;
            carved += bytes;
            return CRISPY_OK;
        }
        CRISPY_TRY(ensure(ctx, own, bytes));
        *out = own.ptr;
        return CRISPY_OK;
    };
    void *keys0, *keys1, *ranges;
    CRISPY_TRY(carve(j.keys, (size_t)m * sizeof(ReadKey), &keys0));
    CRISPY_TRY(carve(j.keys_alt, (size_t)m * sizeof(ReadKey), &keys1));
    CRISPY_TRY(carve(j.range, (size_t)m * sizeof(uint2), &ranges));
    uint2* d_range = static_cast<uint2*>(ranges);
    unsigned long long* d_work = j.counters.as<unsigned long long>() + 4;
    unsigned long long* d_many = d_work + 1;
    const unsigned long long limit = kSettleMost;
    const unsigned blocks = (unsigned)((m + 255) / 256), wblocks = (unsigned)((m + 7) / 8);
    const unsigned tiles = (unsigned)((m + kTile - 1) / kTile);
    ReadKey* ka = nullptr;
    // keys first, reads of equal keys settled group by group; or, where the
    // groups are large (many copies of a read), the reads compared throughout
    auto sort_reads = [&](bool whole) {
        const Ties ties{d_many, whole};
        a = j.idx.as<uint32_t>();
        b = j.idx_alt.as<uint32_t>();
        ka = static_cast<ReadKey*>(keys0);
        ReadKey* kb = static_cast<ReadKey*>(keys1);
        pre_key_kernel<<<blocks, 256, 0, s>>>(rs, a, m, ka);
        pre_sample_kernel<<<1, kSample, 0, s>>>(ka, m, kSettleWorth, d_many);
        count_launch(ctx, 2);
        if (m < 2) return;
        pre_tile_sort_kernel<false><<<tiles, kTileThreads, 0, s>>>(a, ka, m, rs, ties);
        pre_tile_sort_kernel<true><<<tiles, kTileThreads, 0, s>>>(a, ka, m, rs, ties);
        count_launch(ctx, 2);
        for (int64_t w = kTile; w < m; w <<= 1) {
            pre_merge_kernel<<<blocks, 256, 0, s>>>(a, ka, b, kb, m, w, rs, ties);
            count_launch(ctx);
            std::swap(a, b);
            std::swap(ka, kb);
        }
        pre_group_kernel<<<wblocks, 256, 0, s>>>(ka, m, d_range, d_work, ties);
        pre_rank_kernel<<<wblocks, 256, 0, s>>>(a, d_range, m, rs, d_work, limit, b, ties);
        count_launch(ctx, 2);
        std::swap(a, b);
    };
    if (m > 0) {
        sort_reads(false);
        CRISPY_CK(ctx, cudaGetLastError());
    }
    int64_t kept = 0;
    if (m > 0) {
        auto last_of_runs = [&]() -> int {
            pre_last_kernel<<<blocks, 256, 0, s>>>(a, ka, m, rs, j.flags.as<uint8_t>());
            count_launch(ctx);
            CRISPY_CK(ctx, cudaGetLastError());
            return compact_flags(ctx, s, j.flags.as<uint8_t>(), m, j.pos.as<uint32_t>(), j.tiles.as<uint32_t>(),
                                 j.tmp, &kept);
        };
        unsigned long long work = 0;
        CRISPY_CK(ctx, cudaMemcpyAsync(&work, d_work, 8, cudaMemcpyDeviceToHost, s));
        CRISPY_TRY(last_of_runs());   // waits
        if (work > limit) {
            int64_t again = 0;
            CRISPY_TRY(compact_flags(ctx, s, j.alive.as<uint8_t>(), n, j.idx.as<uint32_t>(), j.tiles.as<uint32_t>(),
                                     j.tmp, &again));
            sort_reads(true);
            CRISPY_TRY(last_of_runs());
        }
        pre_emit_kernel<<<(unsigned)((kept + 255) / 256), 256, 0, s>>>(a, j.pos.as<uint32_t>(), kept,
                                                                       j.out_idx.as<int32_t>(),
                                                                       j.out_freq.as<int32_t>());
        count_launch(ctx);
        CRISPY_CK(ctx, cudaGetLastError());
        CRISPY_CK(ctx, cudaMemcpyAsync(out_index, j.out_idx.ptr, (size_t)kept * 4, cudaMemcpyDeviceToHost, s));
        CRISPY_CK(ctx, cudaMemcpyAsync(out_freq, j.out_freq.ptr, (size_t)kept * 4, cudaMemcpyDeviceToHost, s));
    }
    CRISPY_CK(ctx, cudaStreamSynchronize(s));
    j.kept = kept;
    j.n = n;
    j.h_idx.assign(out_index, out_index + kept);
    j.ready = true;
    st.length_discards = (int32_t)(cnt[0] + cnt[1]);
    st.primer_discards = (int32_t)cnt[2];
    st.merges = (int32_t)(m - kept);
    st.kept = (int32_t)kept;
    if (stats) *stats = st;
    return CRISPY_OK;
}
