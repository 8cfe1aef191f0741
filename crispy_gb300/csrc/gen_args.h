// gen_args.h -- launch arguments shared by the genDist DP kernels (gen.cu,
// gen16.cu).  Not part of the public ABI.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>

struct crispy_ctx;

namespace crispy {

struct GenArgs {
    const uint32_t* packed;  // reads, 16 symbols per word, first symbol in the top bits
    const int64_t* woff;     // first packed word of each read
    const int32_t* len;
    const int2* pairs;
    const uint32_t* order;   // optional permutation (length buckets)
    int64_t count;
    int band;
    float* dist;
    int32_t* score;
    int32_t* ml;
    int32_t* al;
    unsigned int* queue;     // optional work counter (persistent launch)
    // 16-bit kernel only: every cell's choice, 2 bits, for the path walk
    // (gen16_dir_words words: one region per pair the grid holds at a
    // time, dir_blocks 16-step blocks long)
    uint32_t* dirs;
    int64_t dirs_words;
    int dir_blocks;
    // 16-bit kernel only: the diagonals each pair is swept over, -lo .. hi as
    // lo | hi << 16 by pair index (nullptr: the whole band), and the pairs
    // whose result that does not prove ([0] their count, then pair indices)
    const uint32_t* bands;
    uint32_t* retry;
    // once more pairs than this are listed, the rest go to the list unswept
    // (0: no limit)
    uint32_t retry_most;
    int ext;                 // pairs beyond kGen16MaxSum: the extended form of the shape
    // All 1.  Adds written as multiply-adds by these run on the FMA pipe;
    // distinct multipliers keep the compiler from factoring a common
    // product back into ALU adds.
    int one[6];
};

// The two-cells-per-register DP (gen16.cu) holds a cell as a 16-bit key
// whose range covers pairs with L1 + L2 <= kGen16MaxSum; longer pairs take
// the 32-bit kernels of gen.cu.
constexpr int kGen16MaxSum = 3600;
// The most L1 + L2 can be: batched runs take longer pairs through the
// extended form first, whose results their scores prove.
constexpr int kGen16ExtSum = 4096;

// Shapes of the 16-bit kernel: G lanes per pair, R registers per lane, so
// a pair swept over diagonals -lo .. hi with (lo + hi) / 2 + 1 <= 2 * G * R
// band slots fits.
struct Shape16 {
    int g, r;
};
int gen16_num_shapes();
Shape16 gen16_shape(int i);
// Pairs per block of a shape (all its warps).
int gen16_pairs_per_block(int i);
// Registers per lane of the shapes a launch of up to `slots` band slots may
// take, up to twice as wide as it needs (bounds the tag storage).
constexpr int gen16_max_r(int slots) { return slots > 256 ? 16 : 8; }
// 16-step blocks a pair's sweep runs at most, for pairs with L1 + L2 <= max_sum.
inline int gen16_dir_blocks(int max_sum) { return (max_sum + 1) / 16 + 1; }
constexpr int kGen16LeanR = 7;   // of the shapes of up to 256 slots
// Words of choice storage a launch of shape i over `count` pairs needs.
int64_t gen16_dir_words(crispy_ctx* ctx, int shape, int64_t count, int dir_blocks, bool ext = false);
// Narrowest shape with an extended form that covers the slots, -1: none.
int gen16_ext_shape(int slots);
// Largest resident threads x registers per lane of one SM over the shapes of
// up to `slots` band slots: a launch holds at most this many tag words per SM
// and sub-block.
int64_t gen16_lane_regs_per_sm(int slots);
// Launch shape i over a.count pairs: persistent grid sized by occupancy.
int gen16_launch(crispy_ctx* ctx, cudaStream_t s, int shape, const GenArgs& a, bool timed);

}  // namespace crispy
