// Time-domain dedispersion with shared channel-group sums: launch interface
// and the sizes the engines need to decide for it and to lay out its rows.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>

#include "tdd_kernels.hpp"

namespace dedisp {
namespace kern {

constexpr int kPatternGroup = 8;  // channels per group
constexpr int kPatternDms = 32;   // DMs per block

struct PatternTotals {
    unsigned long long cost;  // shared-memory wavefronts per tile, all blocks
    unsigned pieces;          // pieces of all blocks
    unsigned rec_words;       // longest record
    unsigned next;            // pieces handed out
    unsigned rows;            // row words of the widest group
    unsigned rounds;          // most rounds of a group
    unsigned pad;             // (the block counts follow, 16-byte aligned)
};

// One piece of a DM block's walk: a channel group, or a round of its trials.
struct PatternPiece {
    int block, group, round;
    int rec_words;           // words kept for its record
    int series, slot;        // first word in the series ring and the row ring
    int series_after;        // pieces of the block that must be summed before
    int slot_after;          // the region is written (-1: none)
    int item;                // building warp of its first run
};

struct PatternTableArgs {
    const float* dms;           // ascending
    int ndm;
    const int32_t* chan_list;   // active channels (delays ascending)
    const float* chan_delay;    // their delays
    int nact;
    int32_t zero_row;           // row index of the all-zero row
    int ngroups;                // (nact + 7) / 8
    int lane_words;             // J
    int period;                 // P of the strided rows, 32 J
    int series_words;           // pattern_series_words
    int series_width;           // pattern_series_width
    int ring_words;             // pattern_ring_words
    int run_words;              // pattern_run_words
    int build_warps;            // pattern_build_warps
    int4* size;                 // [DM blocks][ngroups]
    PatternTotals* totals;
    uint4* block;               // [DM blocks] first piece, pieces; directly behind totals
    // tables proper, sized from the totals
    PatternPiece* sched;        // [pieces]
    uint32_t* rec;              // [pieces][rec_stride]
    size_t rec_stride;          // totals.rec_words
    uint4* win;                 // [pieces][16] copy lists
};
// Sizes (size, block, totals), then the tables.
void launch_pattern_sizes(const PatternTableArgs& a, cudaStream_t s);
void launch_pattern_tables(const PatternTableArgs& a, unsigned pieces, cudaStream_t s);

int tdd_sm_count();  // of the current device

// Words per lane (period P = 32 x that) for a call of `tiles_at_4` blocks at 4
// words per lane, whose widest group stages group_words words beyond the
// periods of its 8 rows; 0 if none fits.
int pattern_lane_words(int nbits, size_t tiles_at_4, long group_words);
int pattern_block_samples(int nbits, int lane_words);  // output samples per block
int pattern_series_words(int nbits);     // positions the series ring holds
int pattern_series_width(int nbits);     // 32-bit words per position
int pattern_ring_words(int nbits);       // words of the row ring
int pattern_run_words(int nbits);        // words a building warp takes at a time
int pattern_build_warps(int nbits, int lane_words);
int pattern_max_group_words(int nbits);  // largest staged rows of a group

// args.tr: strided rows of period 32 x args.lane_words (four byte lanes, or two
// halves for 16-bit input); args.rec/rec_stride/win/block: the tables.
void launch_dedisperse_pattern(const DedisperseArgs& a, cudaStream_t s);
void launch_dedisperse_pattern_batch(const BatchLaunch& b, int nbits, int lane_words, cudaStream_t s);

}  // namespace kern
}  // namespace dedisp
