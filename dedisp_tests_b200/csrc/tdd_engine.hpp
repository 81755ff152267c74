// Execution engine behind TDDPlan and DedispPlan.
//
// One call = validate-free execution of a (sub-)range of the DM list over a
// time series, in gulps of output samples:
//   host rows --(H2D, pinned or pageable)--> gulp input buffer --K1d-->
//   quad-strided rows (pattern and quad kernels; K1: channel-major packed
//   rows for the others) --K2--> output --(D2H)--> host rows. With several gulps, input and
//   output buffers are doubled so that the copies of neighbouring gulps
//   overlap a gulp's kernels; the last gulp's K2 and D2H run per DM group.
// With DEDISP_DEVICE_POINTERS the copies disappear and K1d/K1/K2 read/write
// the caller's buffers. Derived per-plan state (active channels, sorted DMs,
// window sizes) is cached until the DM list or killmask changes.
#pragma once

#include <cstdint>
#include <memory>
#include <vector>

#include "gpu_state.hpp"
#include "tdd_kernels.hpp"
#include "tdd_pattern.hpp"
#include "tdd/TDDPlan.hpp"

namespace dedisp {
namespace detail {

struct TddView {
    size_t nchans;
    const float* delays;
    const int32_t* killmask;
    const float* dms;
    size_t ndm_total;
    size_t max_delay;
    unsigned long version;
};

struct TddCall {
    size_t nsamps;
    const uint8_t* in;
    int in_nbits;
    size_t in_stride;   // bytes
    uint8_t* out;
    int out_nbits;
    size_t out_stride;  // bytes
    size_t first_dm;
    size_t dm_count;
    unsigned flags;
};

// Timing of the last execute() (device time of the dedispersion kernels,
// measured with events on the execution stream; 0 when not recorded).
struct TddStats {
    float kernel_ms = 0.f;
    float transpose_ms = 0.f;
    int launches = 0;
    bool tiled = false;
    int form = -1;       // 0 plain, 1 row by row, 2 shared channel-group sums; -1 none ran
    int lane_words = 0;  // form 2: words per lane
    int rounds = 0;      // form 2: most rounds that a group took its trials in
};

struct TddHostCall;  // model of a host-buffer call (tdd_engine.cpp)

// Whether the pattern kernel takes these (ascending) DMs and active channels'
// delays: it needs ascending delays (no channel of a group is delayed less than
// its first) and sums that its narrow lanes hold.
bool pattern_takes(const std::vector<float>& dms, const std::vector<float>& delays, int nbits);

// The pattern kernel's device tables for one DM list and channel list: size()
// enqueues the size pass for a period, fit() reads its totals and emit()
// enqueues the tables.
class PatternTables {
public:
    // (false: no memory for its sizes)
    bool size(const float* d_dms, size_t ndm, const int32_t* d_chan, const float* d_delay, size_t nact,
              size_t zero_row, int nbits, int lane_words, cudaStream_t st);
    enum Fit { kUse, kRowsFaster, kTooWide };
    // kTooWide: some group's rows do not fit the ring at this period (try a
    // shorter one); kRowsFaster: the row-by-row kernel needs fewer
    // shared-memory wavefronts, or the tables exceed 2 GiB. Waits for `st`.
    Fit fit(cudaStream_t st);
    // Most rounds that a group took its trials in (after fit).
    int rounds() const { return (int)m_total.rounds; }
    // Bytes of the tables that emit() builds (after fit).
    size_t bytes() const;
    // Bytes held for them now.
    size_t held() const { return m_tables.capacity(); }
    // Row words of the widest group beyond its periods (after fit).
    long group_words() const { return (long)m_total.rows - (long)kern::kPatternGroup * 32 * m_args.lane_words; }
    // (false: no memory for the tables, or more than a quarter of what is free:
    // it is left to the rows and outputs)
    bool emit(cudaStream_t st);
    // Table arguments for the DM blocks from `block` on.
    void fill(kern::DedisperseArgs& a, size_t block) const;
    void release();

private:
    rt::DeviceBuffer m_sizes, m_tables;
    kern::PatternTableArgs m_args{};
    kern::PatternTotals m_total{};
    int m_nbits = 0;
};

class TddEngine {
public:
    // Gulp (output samples per pass) unless set: device-resident calls take
    // the largest; calls with host buffers take smaller gulps so that the
    // host copies of neighbouring gulps overlap the kernels.
    static constexpr size_t kDefaultGulp = (size_t)1 << 21;
    static constexpr size_t kHostDefaultGulp = (size_t)1 << 18;

    explicit TddEngine(GpuState& gpu);
    ~TddEngine();

    void execute(const TddView& v, const TddCall& c);

    size_t gulp_size = kDefaultGulp;
    bool gulp_set = false;  // gulp_size was set by the caller
    TddKernel kernel = TddKernel::Auto;
    int variant = -1;  // tile-shape variant of the tiled kernel (8-bit input; -1: default)
    bool record_timing = false;
    bool use_tables = true;   // the pattern kernel may run
    bool keep_form = false;   // the first call of a setup decides the form of all
    TddStats stats;

private:
    struct Setup;
    void prepare(const TddView& v, const TddCall& c);
    void choose_form(const TddView& v, const TddCall& c);
    void choose_gulp(const TddView& v, const TddCall& c, bool shared);
    TddHostCall host_call(const TddView& v, const TddCall& c, bool shared, size_t gulp) const;
    void size_rows(const TddView& v, int nbits);
    // Gives back the tables that the current form does not use; true if there
    // were any.
    bool drop_idle_tables();

    GpuState& m_gpu;
    bool m_pinned = false;  // the current call's host buffers: copies overlap on them
    std::unique_ptr<Setup> m_setup;
    rt::DeviceBuffer m_chan, m_cdl, m_km, m_dms, m_perm, m_tr, m_q, m_out[2], m_stage[2];
    PatternTables m_tables[3];  // 16, 8, 4 words per lane
    rt::PinnedWord m_err_host;
    rt::DeviceBuffer m_err;  // set by a quad-strided kernel whose bounded wait expired
    std::vector<std::unique_ptr<rt::Event>> m_events;
    rt::Event& event(size_t i);
};

}  // namespace detail
}  // namespace dedisp
