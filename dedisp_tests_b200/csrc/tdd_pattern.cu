// Time-domain dedispersion with shared channel-group sums (sm_100a).
//
// Neighbouring trials delay neighbouring channels alike: over a block of 32
// DMs the delays of 8 adjacent channels relative to the first of them take
// only a few distinct patterns (about 9 in a list of 3643 trials over 4096
// channels), because both change by at most a sample or two. The sum of the
// 8 channels under one pattern is the same series for every trial that has
// the pattern, shifted by the trial's delay of the first channel. A block
// therefore builds each pattern's series once in shared memory and every
// trial adds one series per group instead of 8 rows: exact integer sums in a
// different order of additions.
//
// Rows are strided like the quad kernel's (word n of a row holds samples n +
// i*P), so every delay is a whole-word offset. All lanes of a word are summed
// together: S is the plain sum of words, O the sum of the odd lanes moved
// down, and E = S - 2^k O recovers the even lanes at the end (the algebra of
// the 8-bit kernels). Per width:
//   8 bits:  word = 4 samples, series of (S, O) pairs; O and E hold 16-bit
//            lanes, flushed to 32-bit sums every 256 channels
//   <= 4:    word = 4 samples widened to bytes, series of S only (8 x 15 fits
//            a byte), no flush (the engine bounds channels x maximum)
//   16 bits: word = 2 samples, series of (S, O), 32-bit E and O
#include "tdd_pattern.hpp"

#include <algorithm>
#include <type_traits>

#include "runtime.hpp"
#include "tdd_device.cuh"

namespace dedisp {
namespace kern {

int tdd_sm_count()
{
    int dev = 0, sms = 0;
    RT_CHECK(cudaGetDevice(&dev));
    RT_CHECK(cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev));
    return sms;
}

namespace {

constexpr int G = kPatternGroup;    // channels per group
constexpr int D = kPatternDms;      // DMs per block, one lane each in the tables
constexpr int FLUSH_PIECES = 256 / G;
constexpr int LIVE = 8;             // pieces in flight at most (barriers per kind)
constexpr uint32_t FULL = 0xFFFFFFFFu;

// Record of a piece (words), staged in front of its rows
enum {
    REC_LEN = 0,     // words of one series
    REC_WORDS = 1,   // program words
    REC_SERIES = 2,  // byte of the first series in the series ring
    REC_AFTER = 3,   // piece whose series must be summed before this one is built (-1: none)
    REC_ITEM = 4,    // building warp that takes the first run of words
    REC_DM = 8,      // 8 + trial: byte of the trial's sample t0 in the series ring (~0: not in this piece)
    REC_PROG = 40    // program: 8 row offsets (bytes from the record) of the first pattern, then per
                     // change two words: row offset replaced | row offset put in << 16, byte of the
                     // series it is stored to
};
constexpr uint32_t NO_TRIAL = 0xFFFFFFFFu;

enum Mode { kBytes = 0, kByteSums = 1, kHalves = 2 };

// SW: 32-bit words per series position; SPW: samples per word; K: 32-word runs
// a building warp takes at a time. J (a template argument of the kernels) words
// per lane and series make the period P = 32 J. NADD summing warps (warp w
// takes trials w, w + NADD, ..), NBUILD building warps (one more warp stages).
// Registers a thread: REGS at launch; the summing warps, which hold the trials'
// sums, take what the others give up.
template <int MODE> struct Geom;
template <> struct Geom<kBytes>    { static constexpr int SW = 1, SPW = 4, K = 2; };
template <> struct Geom<kByteSums> { static constexpr int SW = 2, SPW = 4, K = 2; };
template <> struct Geom<kHalves>   { static constexpr int SW = 2, SPW = 2, K = 2; };

template <int A, int B, int R, int RA, int RB>
struct WarpSplit
{
    static constexpr int NADD = A, NBUILD = B, TPW = D / A, NT = 32 * (A + B + 1);
    static constexpr int REGS = R, REGS_ADD = RA, REGS_BUILD = RB;
    static_assert(A * RA + (B + 1) * RB <= (A + B + 1) * R, "register split");
};
// Two-word series over 512-word periods leave the summing warps 64 sums and 16
// words in flight each, which takes registers from the building warps. Four
// to eight summing warps left the building ones waiting at 4 bits and less
// (1024 channels, 512 trials: 0.84 ms with 8 + 15, 0.71 with 16 + 11, 0.69 with
// 16 + 15); at 8 bits 8 + 15, 8 + 23 and 16 + 15 took 1.00, 1.04 and 0.93 ms.
template <int MODE, int J>
using Warps = std::conditional_t<(MODE != kBytes && J == 16), WarpSplit<16, 11, 72, 96, 40>, WarpSplit<16, 15, 64, 88, 40>>;

constexpr int mode_of(int nbits) { return nbits == 16 ? kHalves : nbits == 8 ? kByteSums : kBytes; }

// Shared memory: a ring of series and a ring of staged pieces (record and
// rows), both laid out in advance by the tables. At 8 bits 118 KB of series
// hold four pieces of the 3643-trial list's mean (9 patterns of 256 + 135
// words) and 107 KB of rows eight; at 4 bits and less series are half as wide
// and rows (512 + span) words long.
constexpr int kDynBytes = 227 * 1024 - 1024;
__host__ __device__ constexpr int series_bytes(int mode) { return (mode == kBytes ? 92 : 118) * 1024; }
// (512 bytes: a build's last lanes read up to 63 words past a row)
__host__ __device__ constexpr int ring_words(int mode) { return (kDynBytes - 512 - series_bytes(mode)) / 4; }

// odd lanes of a word, moved down
template <int MODE>
__device__ __forceinline__ uint32_t odd_lanes(uint32_t w)
{
    if constexpr (MODE == kHalves) return w >> 16;
    else return __byte_perm(w, 0u, 0x4341);
}

// ---------------------------------------------------------------------------
// Tables. A block walks pieces: its channel groups in order, one piece each; a
// group whose series exceed half the series ring takes its trials in rounds
// of 16, 8 or 4, a piece each.
//   pattern_size_kernel      one warp per (DM block, group), lane = trial
//   pattern_schedule_kernel  one warp per DM block: where each piece's
//                            series and rows lie in the rings and which
//                            earlier piece must be summed first
//   pattern_emit_kernel      one warp per piece: copy list and record
// ---------------------------------------------------------------------------
struct GroupPlan {
    int32_t ch[G];
    int d0, r[G], start4[G], need[G], dst[G];  // dst: words from the group's first row word
    int rows;                                  // row words
    int sub;                                   // trials per round
    uint32_t mine;                             // lanes of this lane's round
    int lo, len, npat;                         // of this lane's round
    bool lead;                                 // lowest lane of its pattern in the round
    int leader, rank, prev;                    // build order; lane of the pattern before
    int cnt;                                   // lead: channels changed (first pattern: 0)
    int changes;                               // of this lane's round
};

__device__ __forceinline__ GroupPlan plan_group(const PatternTableArgs& a, int blk, int group)
{
    GroupPlan p;
    const int lane = threadIdx.x & 31;
    const float dm = a.dms[min(blk * D + lane, a.ndm - 1)];
    uint32_t same = FULL;
    int sum = 0;
#pragma unroll
    for (int c = 0; c < G; ++c) {
        // past the list: the all-zero row at the last channel's delay
        const int j = min(group * G + c, a.nact - 1);
        p.ch[c] = group * G + c < a.nact ? a.chan_list[j] : a.zero_row;
        const int d = (int)delay_rn(dm, a.chan_delay[j]);
        if (c == 0) p.d0 = d;
        p.r[c] = d - p.d0;
        sum += p.r[c];
        same &= __match_any_sync(FULL, p.r[c]);
    }
    const int lo_all = __reduce_min_sync(FULL, p.d0), hi_all = __reduce_max_sync(FULL, p.d0);
    p.rows = 0;
#pragma unroll
    for (int c = 0; c < G; ++c) {
        p.start4[c] = (lo_all + __reduce_min_sync(FULL, p.r[c])) & ~3;
        p.need[c] = (hi_all + __reduce_max_sync(FULL, p.r[c]) + a.period - p.start4[c] + 3) & ~3;
        p.dst[c] = p.rows;
        p.rows += p.need[c];
    }
    // Trials per round: the largest of 32, 16, 8, 4 whose series all fit.
    for (p.sub = D;; p.sub >>= 1) {
        p.mine = p.sub == 32 ? FULL : ((1u << p.sub) - 1u) << (lane & ~(p.sub - 1));
        p.lo = p.d0;
        int hi = p.d0;
        for (int o = p.sub / 2; o > 0; o >>= 1) {
            p.lo = min(p.lo, __shfl_xor_sync(FULL, p.lo, o));
            hi = max(hi, __shfl_xor_sync(FULL, hi, o));
        }
        p.len = hi - p.lo + a.period;
        p.lead = lane == __ffs(same & p.mine) - 1;
        p.npat = __popc(__ballot_sync(FULL, p.lead) & p.mine);
        if (__all_sync(FULL, p.npat * p.len <= a.series_words / 2) || p.sub == 4) break;
    }
    p.leader = __ffs(same & p.mine) - 1;
    const uint32_t leads = __ballot_sync(FULL, p.lead) & p.mine;
    // Build order: from the pattern of least total relative delay, always on
    // to the one that differs in the fewest channels (a tenth to a seventh
    // fewer changes than ascending sums).
    constexpr int NONE = 0x7FFFFFFF;
    p.rank = p.lead ? NONE : 0;
    p.prev = lane;
    p.cnt = 0;
    const int least = __reduce_min_sync(p.mine, p.lead ? sum : NONE);
    int cur = __ffs(__ballot_sync(FULL, p.lead && sum == least) & p.mine) - 1;
    if (lane == cur) p.rank = 0;
    for (int step = 1; step < 32; ++step) {
        int dist = 0;
#pragma unroll
        for (int c = 0; c < G; ++c) dist += __shfl_sync(FULL, p.r[c], cur) != p.r[c];
        const int best = __reduce_min_sync(p.mine, p.lead && p.rank == NONE ? dist * 32 + lane : NONE);
        if (__all_sync(FULL, best == NONE)) break;
        if (best != NONE && lane == (best & 31)) {
            p.rank = step;
            p.prev = cur;
            p.cnt = dist;
        }
        if (best != NONE) cur = best & 31;
    }
    p.changes = 0;
    for (int l = 0; l < 32; ++l) {
        const int n = __shfl_sync(FULL, p.cnt, l);
        if (p.mine >> l & 1u) p.changes += n;
    }
    return p;
}

// 8 row offsets, then two words per change, an even number of changes
__device__ __forceinline__ int program_words(int changes) { return G + 2 * ((changes + 1) & ~1); }

__global__ void __launch_bounds__(128) pattern_size_kernel(PatternTableArgs a)
{
    const int lane = threadIdx.x & 31;
    const int group = blockIdx.x * 4 + (threadIdx.x >> 5), blk = blockIdx.y;
    if (group >= a.ngroups) return;
    const GroupPlan p = plan_group(a, blk, group);
    const int series = __reduce_max_sync(FULL, p.npat * p.len);
    const int len = __reduce_max_sync(FULL, p.len);
    const int rec = REC_PROG + __reduce_max_sync(FULL, program_words(p.changes));
    // Shared-memory wavefronts of this group per tile: the build (8 rows and
    // the program; 2 rows, a quarter program read and a store per change and
    // word) and one series read per trial.
    const int chunks = (p.len + 31) / 32;
    int build = 0;
    if ((lane & (p.sub - 1)) == 0)
        build = chunks * (G + 2 + a.series_width) + chunks * p.changes * (9 + 4 * a.series_width) / 4;
    build = __reduce_add_sync(FULL, build);
    if (lane == 0) {
        const int trials = min(D, a.ndm - blk * D);
        a.size[(size_t)blk * a.ngroups + group] = make_int4(p.rows, series, rec | (p.sub << 16), len);
        atomicAdd(&a.totals->cost, (unsigned long long)(build + trials * (a.period / 32 * a.series_width)));
        atomicAdd(&a.totals->pieces, (unsigned)(D / p.sub));
        atomicMax(&a.totals->rec_words, (unsigned)rec);
        atomicMax(&a.totals->rows, (unsigned)p.rows);
        atomicMax(&a.totals->rounds, (unsigned)(D / p.sub));
        atomicAdd(&a.block[blk].y, (unsigned)(D / p.sub));
    }
}

// One warp per DM block. Both rings are allocated first in, first out; lanes 0..7
// hold where the last eight pieces lie in the series ring, lanes 8..15 in the row
// ring (lane & 7 = piece mod LIVE). A piece is placed behind the one before, or at
// the ring's start where it does not fit, and must wait for the last piece that
// still lies there: `first` is the oldest piece counted live.
//
// Latency bounds it: some twenty dependent steps a piece. One thread per block,
// with the regions in local memory and a load per group, took 5 us a piece: 1.4
// ms for the 192 groups of a beam of 128 trials and 1536 channels, which a batch
// paid for every beam.
__global__ void __launch_bounds__(128) pattern_schedule_kernel(PatternTableArgs a)
{
    static_assert(LIVE == 8, "lanes per ring");
    const int lane = threadIdx.x & 31;
    const int blk = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (blk >= (a.ndm + D - 1) / D) return;
    unsigned base = 0;
    if (lane == 0) {
        const unsigned pieces = a.block[blk].y;
        base = atomicAdd(&a.totals->next, pieces);
        a.block[blk] = make_uint4(base, pieces, 0u, 0u);
    }
    base = __shfl_sync(FULL, base, 0);
    const bool rows = lane >= LIVE;
    const int size = rows ? a.ring_words : a.series_words;
    int head = 0, first = 0;
    int at = 0, len = 0, idx = -1;  // this lane's piece and its region
    int piece = 0, item = 0;
    for (int g0 = 0; g0 < a.ngroups; g0 += 32) {
        int4 mine = make_int4(0, 0, 0, 0);
        if (g0 + lane < a.ngroups) mine = a.size[(size_t)blk * a.ngroups + g0 + lane];
        for (int g = g0; g < min(g0 + 32, a.ngroups); ++g) {
            const int row_words = __shfl_sync(FULL, mine.x, g - g0), series = __shfl_sync(FULL, mine.y, g - g0);
            const int z = __shfl_sync(FULL, mine.z, g - g0), longest = __shfl_sync(FULL, mine.w, g - g0);
            const int rec = z & 0xFFFF, rounds = D / (z >> 16);
            const int n = rows ? rec + row_words : series;
            const int runs = (longest + a.run_words - 1) / a.run_words;
            for (int r = 0; r < rounds; ++r, ++piece) {
                if (head + n > size) head = 0;
                int gone = idx >= first && at < head + n && head < at + len ? idx : -1;
                gone = max(gone, __shfl_xor_sync(FULL, gone, 4));
                gone = max(gone, __shfl_xor_sync(FULL, gone, 2));
                gone = max(gone, __shfl_xor_sync(FULL, gone, 1));
                first = max(first, max(piece - LIVE, gone) + 1);
                if ((lane & (LIVE - 1)) == (piece & (LIVE - 1))) {
                    at = head;
                    len = n;
                    idx = piece;
                }
                const int series_at = __shfl_sync(FULL, head, 0), rows_at = __shfl_sync(FULL, head, LIVE);
                const int series_after = __shfl_sync(FULL, first, 0) - 1, rows_after = __shfl_sync(FULL, first, LIVE) - 1;
                if (lane == 0) {
                    PatternPiece& e = a.sched[base + piece];
                    e.block = blk;
                    e.group = g;
                    e.round = r;
                    e.rec_words = rec;
                    e.series = series_at;
                    e.slot = rows_at;
                    e.series_after = series_after;
                    e.slot_after = rows_after;
                    e.item = item;
                }
                head += n;
                item = (item + runs) % a.build_warps;
            }
        }
    }
}

__global__ void __launch_bounds__(128) pattern_emit_kernel(PatternTableArgs a, unsigned pieces)
{
    const int lane = threadIdx.x & 31;
    const unsigned piece = blockIdx.x * 4 + (threadIdx.x >> 5);
    if (piece >= pieces) return;
    const PatternPiece e = a.sched[piece];
    const GroupPlan p = plan_group(a, e.block, e.group);
    uint32_t* rec = a.rec + (size_t)piece * a.rec_stride;
    uint4* win = a.win + (size_t)piece * 16;

    const bool in = lane / p.sub == e.round;
    const int rlane = e.round * p.sub;  // a lane of the round
    const int len = __shfl_sync(FULL, p.len, rlane), lo = __shfl_sync(FULL, p.lo, rlane);
    const int changes = __shfl_sync(FULL, p.changes, rlane), npat = __shfl_sync(FULL, p.npat, rlane);
    // row offsets of the first pattern, then the changes in build order
    int before = 0;
    for (int l = 0; l < 32; ++l) {
        const int n = __shfl_sync(FULL, p.cnt, l), k = __shfl_sync(FULL, p.rank, l);
        if ((p.mine >> l & 1u) && k < p.rank) before += n;
    }
    uint32_t* prog = rec + REC_PROG;
    uint32_t* out = prog + G + 2 * before;
    const uint32_t series = 4u * (uint32_t)(a.series_width * (e.series + p.rank * len));
#pragma unroll
    for (int c = 0; c < G; ++c) {
        const int rp = __shfl_sync(FULL, p.r[c], p.prev);
        const uint32_t off = 4u * (uint32_t)(e.rec_words + p.dst[c] + lo + p.r[c] - p.start4[c]);
        const uint32_t old = 4u * (uint32_t)(e.rec_words + p.dst[c] + lo + rp - p.start4[c]);
        if (!in || !p.lead) continue;
        if (p.rank == 0) {
            prog[c] = off;
        } else if (rp != p.r[c]) {
            *out++ = old | (off << 16);
            *out++ = series;
        }
    }
    // an odd number of changes: the last pattern again, one word by itself
    if ((changes & 1) && in && p.lead && p.rank == npat - 1) {
        const uint32_t off = 4u * (uint32_t)(e.rec_words + p.dst[0] + lo + p.r[0] - p.start4[0]);
        prog[G + 2 * changes] = off | (off << 16);
        prog[G + 2 * changes + 1] = series;
    }
    const int k = __shfl_sync(FULL, p.rank, p.leader);
    rec[REC_DM + lane] = in ? 4u * (uint32_t)(a.series_width * (e.series + k * len + p.d0 - lo)) : NO_TRIAL;
    if (lane == 0) {
        rec[REC_LEN] = (uint32_t)len;
        rec[REC_WORDS] = (uint32_t)program_words(changes);
        rec[REC_SERIES] = 4u * (uint32_t)(a.series_width * e.series);
        rec[REC_AFTER] = (uint32_t)e.series_after;
        rec[REC_ITEM] = (uint32_t)e.item;
        win[0] = make_uint4(piece, (uint32_t)e.slot_after, (uint32_t)e.rec_words, (uint32_t)e.slot);
    }
#pragma unroll
    for (int c = 0; c < G; ++c)
        if (lane == c)
            win[1 + c] = make_uint4((uint32_t)p.ch[c], (uint32_t)p.start4[c], (uint32_t)p.need[c],
                                    (uint32_t)(e.slot + e.rec_words + p.dst[c]));
}

// ---------------------------------------------------------------------------
// Sums. Block = 32 trials x SPW*P output samples. One warp stages pieces,
// eleven or fifteen build their series, sixteen add them to the trials' sums;
// pieces flow through the two rings, so that no warp waits for the slowest one
// of a step (16 or 32 warps that all built and summed between block barriers
// took 1.25 to 1.48 ms where this takes 0.92: 1024 channels, 512 trials x
// 62914 samples, 8 bits).
//
// Shared-memory wavefronts (68% of peak there, 1500 per piece) and issue slots
// (68%) bound it together: per piece and 32 words of the tile one or two
// wavefronts per trial, and the build's 12 + 2.25 per change + a store per
// pattern. The row-by-row kernel takes one wavefront per trial, channel and 32
// words (2048 per piece), at 84% of peak. Measured, ms, row by row -> here:
// 1024 ch x 512 trials x 62914 samples 1.34 -> 0.92 (8 bits), 0.68 (4 bits);
// 4096 ch x 3643 trials x 95572: 50.6 -> 33.2 (8 bits), 21.1 (2 bits).
// ---------------------------------------------------------------------------
template <int SW>
__device__ __forceinline__ void lds_series(uint32_t addr, uint32_t (&v)[SW])
{
    if constexpr (SW == 2) asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];\n" : "=r"(v[0]), "=r"(v[1]) : "r"(addr));
    else asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v[0]) : "r"(addr));
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr)
{
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];\n" : "=r"(v) : "r"(addr));
    return v;
}
template <int SW>
__device__ __forceinline__ void sts_series(uint32_t addr, uint32_t s, uint32_t o)
{
    if constexpr (SW == 2) asm volatile("st.shared.v2.u32 [%0], {%1, %2};\n" ::"r"(addr), "r"(s), "r"(o) : "memory");
    else asm volatile("st.shared.u32 [%0], %1;\n" ::"r"(addr), "r"(s) : "memory");
}

// 16 words per lane from and to tensor memory (waits for completion)
__device__ __forceinline__ void tmem_ld16(uint32_t addr, uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(addr)
        : "memory");
}
__device__ __forceinline__ void tmem_st16(uint32_t addr, const uint32_t (&v)[16])
{
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};\n\t"
        "tcgen05.wait::st.sync.aligned;" ::"r"(addr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]),
        "r"(v[8]), "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

// Shared state of a tile's warps; barrier p % LIVE of each kind serves piece p.
struct PatternSync {
    uint64_t full[LIVE];    // staged (one arrival, and the copies' bytes)
    uint64_t built[LIVE];   // series built (one arrival per building warp)
    uint64_t summed[LIVE];  // and summed (one per summing warp)
    uint64_t never;         // expiry test: nothing arrives on it
    uint32_t slot[LIVE];    // byte address of the staged record
    int failed;             // a bounded wait expired
    int staged;             // pieces staged
};

__device__ __forceinline__ bool piece_wait(uint64_t* bars, int piece, unsigned long long ns)
{
    return mbar_wait_bounded(&bars[piece & (LIVE - 1)], (uint32_t)(piece / LIVE) & 1u, ns);
}

// The staging warp: lane 0 copies the record, lanes 1..8 the rows.
template <int MODE>
__device__ __forceinline__ void pattern_stage(const DedisperseArgs& a, size_t t0, uint4 blk, uint32_t* smem,
                                              PatternSync& y, WaitCfg wc)
{
    const int lane = threadIdx.x & 31;
    const int pieces = (int)blk.y;
    const uint4* win = a.win + (size_t)blk.x * 16;
    uint32_t* ring = smem + series_bytes(MODE) / 4;
    // copy lists are read two pieces ahead
    uint4 next[2] = {make_uint4(0u, 0u, 0u, 0u), make_uint4(0u, 0u, 0u, 0u)};
#pragma unroll
    for (int i = 0; i < 2; ++i)
        if (i < pieces && lane <= G) next[i] = __ldg(win + (size_t)i * 16 + lane);
    for (int p = 0; p < pieces; ++p) {
        const uint4 c = next[0];
        next[0] = next[1];
        if (p + 2 < pieces && lane <= G) next[1] = __ldg(win + (size_t)(p + 2) * 16 + lane);
        const int after = (int)__shfl_sync(FULL, c.y, 0);
        const uint32_t slot = __shfl_sync(FULL, c.w, 0);
        // addresses before the wait: what follows it is on the chain from one
        // piece's sums to the next piece's rows
        uint64_t* full = &y.full[p & (LIVE - 1)];
        uint32_t n = c.z;
        const uint32_t* src = a.rec + (size_t)c.x * a.rec_stride;
        if (lane > 0) {
            const size_t first = t0 + c.y;
            // windows end inside the row (the pitch leaves room for every
            // trial's reads; what a series may read past them is never used)
            const size_t room = a.tr_pitch_words > first ? a.tr_pitch_words - first : 0;
            if (room < n) n = (uint32_t)room;
            src = a.tr + (size_t)c.x * a.tr_pitch_words + first;
        }
        // (the warp leaves as one: a lane that went on alone would wait for the
        // others in the next shuffle for good)
        if (after >= 0 && !__all_sync(FULL, piece_wait(y.summed, after, wc.ns))) {
            if (lane == 0) atomicExch(&y.failed, 1);
            return;
        }
        if (lane <= G && n) {
            mbar_expect_tx(full, 4u * n);
            bulk_g2s(ring + c.w, src, 4u * n, full);
        }
        if (lane == 0) {
            y.slot[p & (LIVE - 1)] = smem_addr(ring + slot);
            y.staged = p + 1;
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(full);
    }
}

// The building warps. Runs of 32 K words of the pieces' series are dealt to
// the warps in turn, across pieces.
template <int MODE, int J>
__device__ __forceinline__ void pattern_build(uint4 blk, uint32_t series, PatternSync& y, WaitCfg wc)
{
    constexpr int SW = Geom<MODE>::SW, K = Geom<MODE>::K, NADD = Warps<MODE, J>::NADD, NBUILD = Warps<MODE, J>::NBUILD;
    const int lane = threadIdx.x & 31, bw = (int)(threadIdx.x >> 5) - NADD;
    const int pieces = (int)blk.y;
    for (int p = 0; p < pieces; ++p) {
        bool ok = piece_wait(y.full, p, wc.ns);
        // expiry test: one more wait, on a barrier nothing arrives on
        if (wc.expiry_test && p == 0) ok = ok && mbar_wait_bounded(&y.never, 0u, wc.ns);
        const uint32_t slot = *(volatile uint32_t*)&y.slot[p & (LIVE - 1)];
        if (ok) {
            const int after = (int)lds32(slot + 4u * REC_AFTER);
            if (after >= 0) ok = piece_wait(y.summed, after, wc.ns);
        }
        if (!__all_sync(FULL, ok)) {
            if (lane == 0) atomicExch(&y.failed, 1);
            return;
        }
        const uint4 h = lds128(slot);
        const int len = (int)h.x;
        const uint32_t prog = slot + 4u * REC_PROG, prog_end = prog + 4u * h.y;
        int run = bw - (int)lds32(slot + 4u * REC_ITEM);
        if (run < 0) run += NBUILD;
        for (int n = 32 * K * run + lane; n - lane < len; n += 32 * K * NBUILD) {
            const uint32_t rows = slot + 4u * (uint32_t)n;
            const uint32_t to = series + 4u * SW * (uint32_t)n;
            bool keep[K];
            uint32_t s[K], o[K];
            const uint4 e0 = lds128(prog), e1 = lds128(prog + 16u);
            uint4 c = lds128(prog + 32u);  // the first two changes
            {
                const uint32_t e[8] = {e0.x, e0.y, e0.z, e0.w, e1.x, e1.y, e1.z, e1.w};
                uint32_t x[8][K];
#pragma unroll
                for (int i = 0; i < 8; ++i)
#pragma unroll
                    for (int k = 0; k < K; ++k) x[i][k] = lds32(rows + e[i] + 128u * k);
#pragma unroll
                for (int k = 0; k < K; ++k) {
                    keep[k] = n + 32 * k < len;
                    s[k] = o[k] = 0;
#pragma unroll
                    for (int i = 0; i < 8; ++i) {
                        s[k] += x[i][k];
                        if constexpr (SW == 2) o[k] += odd_lanes<MODE>(x[i][k]);
                    }
                    if (keep[k]) sts_series<SW>(to + h.z + 128u * SW * k, s[k], o[k]);
                }
            }
            for (uint32_t q = prog + 32u; q < prog_end; q += 16u) {
                const uint4 now = c;
                c = lds128(q + 16u);  // the next two (unused past the last)
                const uint32_t at[4] = {rows + (now.x & 0xFFFFu), rows + (now.x >> 16), rows + (now.z & 0xFFFFu),
                                        rows + (now.z >> 16)};
                uint32_t v[4][K];
#pragma unroll
                for (int i = 0; i < 4; ++i)
#pragma unroll
                    for (int k = 0; k < K; ++k) v[i][k] = lds32(at[i] + 128u * k);
#pragma unroll
                for (int i = 0; i < 2; ++i)
#pragma unroll
                    for (int k = 0; k < K; ++k) {
                        s[k] = s[k] + v[2 * i + 1][k] - v[2 * i][k];
                        if constexpr (SW == 2)
                            o[k] = o[k] + odd_lanes<MODE>(v[2 * i + 1][k]) - odd_lanes<MODE>(v[2 * i][k]);
                        if (keep[k]) sts_series<SW>(to + (i ? now.w : now.y) + 128u * SW * k, s[k], o[k]);
                    }
            }
        }
        __syncwarp();
        if (lane == 0) mbar_arrive(&y.built[p & (LIVE - 1)]);
    }
}

template <int MODE, int J>
__device__ __forceinline__ void pattern_tile(const DedisperseArgs& a, int bx, size_t by, uint32_t tmem, WaitCfg wc)
{
    constexpr int SW = Geom<MODE>::SW, SPW = Geom<MODE>::SPW;
    constexpr int NADD = Warps<MODE, J>::NADD, NBUILD = Warps<MODE, J>::NBUILD, TPW = Warps<MODE, J>::TPW;
    constexpr int P = 32 * J;
    constexpr size_t BT = (size_t)SPW * P;

    extern __shared__ __align__(128) uint32_t smem[];
    __shared__ PatternSync y;

    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const size_t t0 = by * BT;
    const int i0 = bx * D;
    const int nvalid = min(D, a.ndm - i0);
    const uint4 blk = a.block[bx];
    const int pieces = (int)blk.y;
    const uint32_t series = smem_addr(smem);

    if (threadIdx.x == 0) {
        for (int i = 0; i < LIVE; ++i) {
            mbar_init(&y.full[i], 1);
            mbar_init(&y.built[i], NBUILD);
            mbar_init(&y.summed[i], NADD);
        }
        mbar_init(&y.never, 1);
        y.failed = 0;
        y.staged = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();

    if (warp >= NADD) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Warps<MODE, J>::REGS_BUILD));
        if (warp == NADD + NBUILD) pattern_stage<MODE>(a, t0, blk, smem, y, wc);
        else pattern_build<MODE, J>(blk, series, y, wc);
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Warps<MODE, J>::REGS));
    } else {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(Warps<MODE, J>::REGS_ADD));
        uint32_t S[TPW][J], O[TPW][J];
#pragma unroll
        for (int h = 0; h < TPW; ++h)
#pragma unroll
            for (int k = 0; k < J; ++k) S[h][k] = O[h][k] = 0;
        // 8 bits: 32-bit sums of 4 lane words (16 samples) from k0 on, from the
        // 16-bit lanes and, unless `first`, the sums so far. Those are kept in
        // tensor memory, 4 J columns a trial: they would take half of the
        // registers.
        const uint32_t tsum = tmem + ((uint32_t)(warp & 3) << 21) + (uint32_t)(warp >> 2) * (4 * TPW * J);
        auto wide_sums = [&](int h, int k0, bool first, uint32_t (&sum)[16]) {
            if (first) {
#pragma unroll
                for (int k = 0; k < 16; ++k) sum[k] = 0;
            } else {
                tmem_ld16(tsum + (uint32_t)(4 * (h * J + k0)), sum);
            }
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t o = O[h][k0 + k], e = S[h][k0 + k] - 256u * o;
                sum[4 * k + 0] += e & 0xFFFFu;
                sum[4 * k + 2] += e >> 16;
                sum[4 * k + 1] += o & 0xFFFFu;
                sum[4 * k + 3] += o >> 16;
                S[h][k0 + k] = O[h][k0 + k] = 0;
            }
        };

        int since_flush = 0;  // pieces summed since the last flush
        bool flushed = false, ok = true;
        for (int p = 0; p < pieces; ++p) {
            ok = piece_wait(y.built, p, wc.ns);
            if (!__all_sync(FULL, ok)) {
                if (lane == 0) atomicExch(&y.failed, 1);
                break;
            }
            const uint32_t slot = *(volatile uint32_t*)&y.slot[p & (LIVE - 1)];
            uint32_t at[TPW];
#pragma unroll
            for (int h = 0; h < TPW; ++h) at[h] = lds32(slot + 4u * (uint32_t)(REC_DM + warp + NADD * h));
            if (MODE == kByteSums && since_flush == FLUSH_PIECES) {
#pragma unroll
                for (int h = 0; h < TPW; ++h)
#pragma unroll
                    for (int k0 = 0; k0 < J; k0 += 4) {
                        uint32_t sum[16];
                        wide_sums(h, k0, !flushed, sum);
                        tmem_st16(tsum + (uint32_t)(4 * (h * J + k0)), sum);
                    }
                flushed = true;
                since_flush = 0;
            }
            ++since_flush;
#pragma unroll
            for (int h = 0; h < TPW; ++h) {
                if (warp + NADD * h >= nvalid || at[h] == NO_TRIAL) continue;
                const uint32_t from = series + at[h] + 4u * SW * (uint32_t)lane;
                constexpr int KB = J < 8 ? J : 8;  // words per lane loaded at a time
#pragma unroll
                for (int k0 = 0; k0 < J; k0 += KB) {
                    uint32_t v[KB][SW];
#pragma unroll
                    for (int k = 0; k < KB; ++k) lds_series<SW>(from + 128u * SW * (uint32_t)(k0 + k), v[k]);
#pragma unroll
                    for (int k = 0; k < KB; ++k) {
                        S[h][k0 + k] += v[k][0];
                        if constexpr (SW == 2) O[h][k0 + k] += v[k][1];
                        else O[h][k0 + k] += odd_lanes<MODE>(v[k][0]);
                    }
                }
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&y.summed[p & (LIVE - 1)]);
        }
        ok = __all_sync(FULL, ok);
#pragma unroll
        for (int h = 0; h < TPW; ++h) {
            const int trial = warp + NADD * h;
            if (!ok || trial >= nvalid) continue;
            const int row = a.perm ? a.perm[i0 + trial] : i0 + trial;
            const size_t base = (size_t)row * a.out_stride;
#pragma unroll
            for (int k0 = 0; k0 < J; k0 += 4) {
                uint32_t sum[16];
                if constexpr (MODE == kByteSums) {
                    wide_sums(h, k0, !flushed, sum);
                } else {
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        const uint32_t o = O[h][k0 + k];
                        if constexpr (MODE == kBytes) {
                            const uint32_t e = S[h][k0 + k] - 256u * o;
                            sum[4 * k + 0] = e & 0xFFFFu;
                            sum[4 * k + 1] = o & 0xFFFFu;
                            sum[4 * k + 2] = e >> 16;
                            sum[4 * k + 3] = o >> 16;
                        } else {
                            sum[4 * k + 0] = S[h][k0 + k] - 65536u * o;
                            sum[4 * k + 1] = o;
                        }
                    }
                }
#pragma unroll
                for (int k = 0; k < 4; ++k)
#pragma unroll
                    for (int i = 0; i < SPW; ++i) {
                        const size_t t = t0 + (size_t)(lane + 32 * (k0 + k)) + (size_t)i * P;
                        if (t < a.nsamp_out)
                            store_out(a.out, base + t, a.out_nbits, sum[4 * k + i], a.den, a.factor);
                    }
            }
        }
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(Warps<MODE, J>::REGS));
    }
    // the barriers are initialised afresh by the next tile of a persistent block
    __syncthreads();
    if (threadIdx.x == 0) {
        if (y.failed) {
            // wait (bounded) for the copies in flight and record the error
            for (int p = max(0, y.staged - LIVE); p < y.staged; ++p) piece_wait(y.full, p, wc.ns);
            atomicExch(a.err, 1u);
        }
        for (int i = 0; i < LIVE; ++i) {
            mbar_inval(&y.full[i]);
            mbar_inval(&y.built[i]);
            mbar_inval(&y.summed[i]);
        }
        mbar_inval(&y.never);
    }
    __syncthreads();
}

// Tensor memory of a block's 32-bit sums (8 bits): 16 warps of 32 lanes x 2
// trials x 4 J words, 32 J of the 512 columns. Returns its address; every thread
// calls it.
template <int MODE, int J>
__device__ __forceinline__ uint32_t sums_alloc()
{
    __shared__ uint32_t s_tmem;
    if constexpr (MODE == kByteSums) {
        if (threadIdx.x < 32) {
            asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(&s_tmem)),
                         "n"(32 * J)
                         : "memory");
            asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
        }
        __syncthreads();
        return s_tmem;
    }
    return 0u;
}
template <int MODE, int J>
__device__ __forceinline__ void sums_free(uint32_t tmem)
{
    if constexpr (MODE == kByteSums) {
        __syncthreads();
        if (threadIdx.x < 32)
            asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "n"(32 * J));
    }
}

template <int MODE, int J>
__global__ void __launch_bounds__(Warps<MODE, J>::NT, 1) dedisperse_pattern_kernel(DedisperseArgs a, WaitCfg wc)
{
    const uint32_t tmem = sums_alloc<MODE, J>();
    pattern_tile<MODE, J>(a, blockIdx.x, blockIdx.y, tmem, wc);
    sums_free<MODE, J>(tmem);
}

template <int MODE, int J>
__global__ void __launch_bounds__(Warps<MODE, J>::NT, 1)
dedisperse_pattern_batch_kernel(const DedisperseArgs* __restrict__ args,
                                const unsigned long long* __restrict__ item_start,
                                const int* __restrict__ nbx, int nbeams, WaitCfg wc)
{
    const uint32_t tmem = sums_alloc<MODE, J>();
    batch_items(args, item_start, nbx, nbeams,
                [&](const DedisperseArgs& a, int bx, size_t by) { pattern_tile<MODE, J>(a, bx, by, tmem, wc); });
    sums_free<MODE, J>(tmem);
}

template <int MODE, int J>
void launch_shape(const DedisperseArgs& a, cudaStream_t s)
{
    auto kfn = dedisperse_pattern_kernel<MODE, J>;
    rt::raise_smem_limit(kfn, kDynBytes);
    const size_t bt = (size_t)(32 * J * Geom<MODE>::SPW);
    dim3 grid((a.ndm + D - 1) / D, (unsigned)((a.nsamp_out + bt - 1) / bt));
    kfn<<<grid, Warps<MODE, J>::NT, kDynBytes, s>>>(a, wait_cfg());
    RT_CHECK(cudaGetLastError());
}

template <int MODE, int J>
void launch_batch_shape(const BatchLaunch& b, cudaStream_t s)
{
    auto kfn = dedisperse_pattern_batch_kernel<MODE, J>;
    rt::raise_smem_limit(kfn, kDynBytes);
    const unsigned grid =
        (unsigned)std::max<unsigned long long>(1, std::min<unsigned long long>(tdd_sm_count(), b.total_items));
    kfn<<<grid, Warps<MODE, J>::NT, kDynBytes, s>>>(b.args, b.item_start, b.nbx, b.nbeams, wait_cfg());
    RT_CHECK(cudaGetLastError());
}

template <int MODE>
void launch_mode(const DedisperseArgs& a, cudaStream_t s)
{
    switch (a.lane_words) {
    case 4: launch_shape<MODE, 4>(a, s); break;
    case 8: launch_shape<MODE, 8>(a, s); break;
    case 16: launch_shape<MODE, 16>(a, s); break;
    default: DD_THROW_MSG(DEDISP_INTERNAL_GPU_ERROR, "unknown pattern kernel shape");
    }
}

template <int MODE>
void launch_batch_mode(const BatchLaunch& b, int lane_words, cudaStream_t s)
{
    switch (lane_words) {
    case 4: launch_batch_shape<MODE, 4>(b, s); break;
    case 8: launch_batch_shape<MODE, 8>(b, s); break;
    case 16: launch_batch_shape<MODE, 16>(b, s); break;
    default: DD_THROW_MSG(DEDISP_INTERNAL_GPU_ERROR, "unknown pattern kernel shape");
    }
}

template <int MODE>
int build_warps(int lane_words)
{
    return lane_words == 16 ? Warps<MODE, 16>::NBUILD : lane_words == 8 ? Warps<MODE, 8>::NBUILD : Warps<MODE, 4>::NBUILD;
}

}  // namespace

// Long periods build fewer words past their samples (a window is P + span
// words) and spread a piece's fixed costs, short ones fill the chip: the least
// of waves x (J + c), the time of a tile in units of its words. c from 1024
// channels x 512 trials x 62914 samples, 3.4 waves at J = 16 and 6.7 at J = 8
// (8 bits 1.04 and 0.92 ms, 4 bits 0.68 and 0.78 ms) and 4096 channels x 3643
// trials x 95572 samples, 36 and 72 waves (8 bits 33.2 and 35.8 ms).
int pattern_lane_words(int nbits, size_t tiles_at_4, long group_words)
{
    const size_t sms = (size_t)tdd_sm_count();
    const int c = mode_of(nbits) == kBytes ? 6 : 1;
    int best = 0;
    size_t least = 0;
    for (int j : {16, 8, 4}) {
        if (group_words + (long)(G * 32 * j) > pattern_max_group_words(nbits)) continue;
        const size_t tiles = (tiles_at_4 * 4 + j - 1) / j;
        const size_t cost = (tiles + sms - 1) / sms * (size_t)(j + c);
        if (!best || cost < least) {
            best = j;
            least = cost;
        }
    }
    return best;
}

int pattern_block_samples(int nbits, int lane_words) { return 32 * lane_words * (nbits == 16 ? 2 : 4); }
int pattern_series_words(int nbits)
{
    const int m = mode_of(nbits);
    return series_bytes(m) / (m == kBytes ? 4 : 8);
}
int pattern_series_width(int nbits) { return mode_of(nbits) == kBytes ? 1 : 2; }
int pattern_ring_words(int nbits) { return ring_words(mode_of(nbits)); }
int pattern_run_words(int nbits) { return 32 * (mode_of(nbits) == kBytes ? Geom<kBytes>::K : Geom<kByteSums>::K); }
int pattern_build_warps(int nbits, int lane_words)
{
    switch (mode_of(nbits)) {
    case kBytes: return build_warps<kBytes>(lane_words);
    case kByteSums: return build_warps<kByteSums>(lane_words);
    default: return build_warps<kHalves>(lane_words);
    }
}
// A piece (record: at most 8 + 2 x 32 x 7 program words) takes at most half of
// the ring, and its row offsets are bytes below 2^16.
int pattern_max_group_words(int nbits)
{
    return std::min(pattern_ring_words(nbits) / 2, 16380) - REC_PROG - (G + 2 * 32 * 7) - 4;
}

void launch_pattern_sizes(const PatternTableArgs& a, cudaStream_t s)
{
    const unsigned nblk = (unsigned)((a.ndm + D - 1) / D);
    if (nblk > 65535u) DD_THROW_MSG(DEDISP_UNKNOWN_ERROR, "too many DM blocks for one table launch");
    // the block counts follow the totals
    RT_CHECK(cudaMemsetAsync(a.totals, 0, sizeof(PatternTotals) + nblk * sizeof(uint4), s));
    pattern_size_kernel<<<dim3((unsigned)((a.ngroups + 3) / 4), nblk), 128, 0, s>>>(a);
    RT_CHECK(cudaGetLastError());
}

void launch_pattern_tables(const PatternTableArgs& a, unsigned pieces, cudaStream_t s)
{
    const unsigned nblk = (unsigned)((a.ndm + D - 1) / D);
    pattern_schedule_kernel<<<(nblk + 3) / 4, 128, 0, s>>>(a);
    RT_CHECK(cudaGetLastError());
    pattern_emit_kernel<<<(pieces + 3) / 4, 128, 0, s>>>(a, pieces);
    RT_CHECK(cudaGetLastError());
}

void launch_dedisperse_pattern(const DedisperseArgs& a, cudaStream_t s)
{
    if (a.err == nullptr || a.rec == nullptr || a.win == nullptr || a.block == nullptr)
        DD_THROW_MSG(DEDISP_INTERNAL_GPU_ERROR, "pattern launch without its tables");
    switch (mode_of(a.nbits)) {
    case kBytes: launch_mode<kBytes>(a, s); break;
    case kByteSums: launch_mode<kByteSums>(a, s); break;
    default: launch_mode<kHalves>(a, s); break;
    }
}

void launch_dedisperse_pattern_batch(const BatchLaunch& b, int nbits, int lane_words, cudaStream_t s)
{
    if (b.total_items == 0) return;
    switch (mode_of(nbits)) {
    case kBytes: launch_batch_mode<kBytes>(b, lane_words, s); break;
    case kByteSums: launch_batch_mode<kByteSums>(b, lane_words, s); break;
    default: launch_batch_mode<kHalves>(b, lane_words, s); break;
    }
}

}  // namespace kern
}  // namespace dedisp
