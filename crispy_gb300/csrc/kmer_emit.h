// kmer_emit.h -- device helpers shared by the k-mer kernels (kmer.cu,
// kmer_filter.cu): stage order keys and survivor emission.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

namespace crispy {
namespace {

// Bits of 0 .. v - 1.
__host__ __device__ __forceinline__ int index_bits(int v) {
    int b = 0;
    while (b < 31 && (1 << b) < v) ++b;
    return b;
}

// kmerCUDA.cu:79-111 + Trag_reverse_eq (kmerMain.cpp:205-216): stages
// enumerate the upper triangle of the stageDim grid row-major; inside a stage
// the host scan is row-major (kmerMain.cpp:175-195).  The key holds stage row,
// stage column, row and column inside the stage, from the top, each in as
// many bits as it needs: 36 bits at 100,000 reads, 42 at the most.
__device__ __forceinline__ uint64_t stage_key(int r, int c, int A, int sd) {
    const int ab = 32 - __clz(A - 1), sb = sd > 1 ? 32 - __clz(sd - 1) : 0;
    const int sx = r / A, sy = c / A;
    return ((((uint64_t)sx << sb) | (uint64_t)sy) << (2 * ab)) | ((uint64_t)(r - sx * A) << ab) |
           (uint64_t)(c - sy * A);
}
__device__ __forceinline__ int2 stage_pair(uint64_t key, int A, int sd) {
    const int ab = 32 - __clz(A - 1), sb = sd > 1 ? 32 - __clz(sd - 1) : 0;
    const uint32_t am = (1u << ab) - 1u, sm = (1u << sb) - 1u;
    return make_int2((int)(key >> (2 * ab + sb)) * A + (int)((uint32_t)(key >> ab) & am),
                     (int)((uint32_t)(key >> (2 * ab)) & sm) * A + (int)((uint32_t)key & am));
}
inline int stage_key_bits(int A, int sd) { return 2 * index_bits(A) + 2 * index_bits(sd); }

// Survivor emission with one atomic per warp.  All 32 lanes call it.
// (r, c) are positions in the job's read order; with a read order (perm !=
// nullptr, K = 8) they map back to the caller's read IDs, the pair is
// reordered so that the lower ID comes first, and only pairs whose lower ID
// lies in [olo, ohi) are kept (the stage rows of one pass).
__device__ __forceinline__ void emit(unsigned long long* counter, uint64_t* keys, uint32_t* vals,
                                     int64_t cap, int A, int sd, const int32_t* perm,
                                     int olo, int ohi, bool pass, int r, int c, int m, int mn,
                                     int base_pos = 0, uint64_t tag = 0, unsigned long long* jcount = nullptr) {
    if (perm != nullptr && pass) {
        const int pr = __ldg(perm + r), pc = __ldg(perm + c);
        r = min(pr, pc);
        c = max(pr, pc);
        pass = r >= olo && r < ohi;
    }
    const unsigned pm = __ballot_sync(0xffffffffu, pass);
    if (!pm) return;
    const int lane = threadIdx.x & 31;
    unsigned long long base = 0;
    const int leader = __ffs(pm) - 1;
    if (lane == leader) {
        base = atomicAdd(counter, (unsigned long long)__popc(pm));
        if (jcount) atomicAdd(jcount, (unsigned long long)__popc(pm));
    }
    base = __shfl_sync(0xffffffffu, base, leader);
    if (pass) {
        const unsigned long long idx = base + __popc(pm & ((1u << lane) - 1u));
        if (idx < (unsigned long long)cap) {
            keys[idx] = tag | stage_key(r - base_pos, c - base_pos, A, sd);
            // kmerKernel.cu:47: 1.0f - (float)matches / min(T1, T2), IEEE
            const float d = __fsub_rn(1.0f, __fdiv_rn((float)m, (float)mn));
            vals[idx] = __float_as_uint(d);
        }
    }
}

}  // namespace
}  // namespace crispy
