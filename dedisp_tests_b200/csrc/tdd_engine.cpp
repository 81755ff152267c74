// TDD execution engine (see tdd_engine.hpp).
#include "tdd_engine.hpp"

#include <algorithm>
#include <cmath>
#include <numeric>

#include "host_math.hpp"
#include "tdd_kernels.hpp"
#include "tdd_pattern.hpp"

namespace dedisp {
namespace detail {

namespace {
constexpr int kMaxOutGroups = 8;                   // DM groups for D2H overlap
// A DM range, mask or width that is new to the plan costs the shared sums 0.1 to
// 0.3 ms of tables, and where they decline 0.1 ms to know it. From about 2e9
// additions (trials x channels x samples, 0.2 ms row by row) one call earns that
// back; a smaller one runs row by row and leaves the tables to the next call on
// the same setup. Calls alternating over two ranges, ms, tables at once against
// none: 64 channels x 32 trials x 8192 samples 0.117 and 0.092, 256 x 32 x 16384
// (declined) 0.25 and 0.136, 1024 x 32 x 62914 0.355 and 0.385, 1024 x 512 x
// 62914 1.06 and 1.72.
constexpr double kTablesAtOnce = 2e9;

size_t round_up(size_t a, size_t b) { return (a + b - 1) / b * b; }
int table_index(int lane_words) { return lane_words == 16 ? 0 : lane_words == 8 ? 1 : 2; }
}  // namespace

bool pattern_takes(const std::vector<float>& dms, const std::vector<float>& delays, int nbits)
{
    const size_t nact = delays.size();
    if (nbits > 16 || nact == 0 || dms.empty()) return false;
    if (nbits < 8 && nact * ((1u << nbits) - 1u) > 65535u) return false;  // 16-bit lanes
    if (nbits == 16 && nact > 65536u) return false;                       // 32-bit sums
    if (!(delays.front() >= 0.f) || !std::is_sorted(delays.begin(), delays.end())) return false;
    if ((dms.size() + kern::kPatternDms - 1) / kern::kPatternDms > 65535) return false;
    // (the tables add up 8 rows and 32 series of the delays' span in 32 bits)
    return hostmath::delay_rn(dms.back(), delays.back()) < (1u << 25);
}

// Everything derived from (DM list, killmask, DM range, nbits, kernel choice).
struct TddEngine::Setup {
    unsigned long version = ~0ul;
    size_t first = ~(size_t)0, count = ~(size_t)0;
    int nbits = -1;
    TddKernel kernel = TddKernel::Auto;
    int variant = -1;

    bool tiled_ok = false;       // a tiled form may run (0/1 killmask, not plain by choice)
    bool pattern_ok = false;     // and the pattern kernel among them
    long group_words = 0;        // widest group's row words beyond its periods (0: not known yet)
    int table[3] = {0, 0, 0};    // pattern tables for 16, 8, 4 words per lane: 1 built, -1 rows are faster
    bool rows_sized = false;     // row-by-row form: sizes below are set
    bool rows_tiled = false, rows_quad = false;
    int rows_period = 0;

    // form of the current call
    size_t gulp = 0;             // output samples per pass
    bool form_chosen = false;
    bool tables_due = false;     // row by row for now, the tables at a later call
    bool tiled = false;
    bool quad = false;           // strided rows (quad kernels, pattern kernel)
    bool pattern = false;        // shared channel-group sums (tdd_pattern.hpp)
    int lane_words = 0;          // pattern: words per lane
    int period = 0;              // strided rows: P, words per lane set
    int nact = 0;
    int win_words = 0;
    int chan_per_stage = 0;
    int nstages = 0;
    uint32_t tmax = 0;           // largest delay of the range over active channels
    bool identity = true;        // DM range already ascending
    std::vector<int32_t> chan_list;
    std::vector<uint32_t> km_vals;
    std::vector<float> dms;      // ascending (tiled) or in list order (plain)
    std::vector<int32_t> perm;   // output row of each slot
};

bool PatternTables::size(const float* d_dms, size_t ndm, const int32_t* d_chan, const float* d_delay, size_t nact,
                         size_t zero_row, int nbits, int lane_words, cudaStream_t st)
{
    const size_t nblk = (ndm + kern::kPatternDms - 1) / kern::kPatternDms;
    const size_t ngroups = (nact + kern::kPatternGroup - 1) / kern::kPatternGroup;
    const size_t head = sizeof(kern::PatternTotals) + nblk * sizeof(uint4);
    static_assert(sizeof(kern::PatternTotals) % sizeof(uint4) == 0, "block counts follow the totals");
    if (!m_sizes.reserve_optional(head + nblk * ngroups * sizeof(int4))) return false;
    m_nbits = nbits;
    kern::PatternTableArgs a{};
    a.dms = d_dms;
    a.ndm = (int)ndm;
    a.chan_list = d_chan;
    a.chan_delay = d_delay;
    a.nact = (int)nact;
    a.zero_row = (int32_t)zero_row;
    a.ngroups = (int)ngroups;
    a.lane_words = lane_words;
    a.period = 32 * lane_words;
    a.series_words = kern::pattern_series_words(nbits);
    a.series_width = kern::pattern_series_width(nbits);
    a.ring_words = kern::pattern_ring_words(nbits);
    a.run_words = kern::pattern_run_words(nbits);
    a.build_warps = kern::pattern_build_warps(nbits, lane_words);
    uint8_t* base = m_sizes.get<uint8_t>();
    a.totals = reinterpret_cast<kern::PatternTotals*>(base);
    a.block = reinterpret_cast<uint4*>(base + sizeof(kern::PatternTotals));
    a.size = reinterpret_cast<int4*>(base + head);
    kern::launch_pattern_sizes(a, st);
    m_args = a;
    return true;
}

PatternTables::Fit PatternTables::fit(cudaStream_t st)
{
    RT_CHECK(cudaMemcpyAsync(&m_total, m_args.totals, sizeof(m_total), cudaMemcpyDeviceToHost, st));
    RT_CHECK(cudaStreamSynchronize(st));
    if ((long)m_total.rows > kern::pattern_max_group_words(m_nbits)) return kTooWide;
    // Wavefronts of the row-by-row kernel over the same tiles: one per trial,
    // channel and 32 words, at a higher rate (256 channels, 512 trials 10
    // samples apart, 2 bits: 0.240 ms here against 0.231 at nearly equal
    // wavefronts; 5% below them the two are even).
    const unsigned long long rows = (unsigned long long)m_args.ndm * m_args.nact * m_args.lane_words;
    return m_total.cost * 8 >= rows * 7 || bytes() > ((size_t)2 << 30) ? kRowsFaster : kUse;
}

size_t PatternTables::bytes() const
{
    return m_total.pieces * (sizeof(kern::PatternPiece) + 16 * sizeof(uint4) + (size_t)m_total.rec_words * 4);
}

void PatternTables::release()
{
    m_sizes.release();
    m_tables.release();
}

bool PatternTables::emit(cudaStream_t st)
{
    kern::PatternTableArgs& a = m_args;
    const size_t n = m_total.pieces;
    a.rec_stride = m_total.rec_words;
    const size_t win = n * 16 * sizeof(uint4), rec = n * a.rec_stride * 4;  // 16-byte multiples
    if (!m_tables.reserve_optional(bytes())) return false;
    uint8_t* base = m_tables.get<uint8_t>();
    a.win = reinterpret_cast<uint4*>(base);
    a.rec = reinterpret_cast<uint32_t*>(base + win);
    a.sched = reinterpret_cast<kern::PatternPiece*>(base + win + rec);
    kern::launch_pattern_tables(a, m_total.pieces, st);
    return true;
}

void PatternTables::fill(kern::DedisperseArgs& a, size_t block) const
{
    a.rec = m_args.rec;
    a.rec_stride = m_args.rec_stride;
    a.win = m_args.win;
    a.block = m_args.block + block;
    a.lane_words = m_args.lane_words;
}

// Host-buffer calls: time of a pass over the output samples, from the copies and
// the tiles of a form.
struct TddHostCall {
    size_t nout, ndm, tmax;      // output samples, trials, largest delay
    size_t row_bytes, out_bytes; // of an input row, of an output sample of all trials
    size_t nchans;
    bool identity;               // output rows in the order of the trials
    size_t block_samples, block_dms;
    double tile_us;              // one tile
    size_t sms;
    double copy_rate;            // bytes per us, either way
};

namespace {
// Rates of a B200 on its host's bus: pinned buffers 52 GB/s either way, 72 both
// ways together, pageable ones 10; the kernels' rows are made at 3 TB/s.
constexpr double kPinnedBytesPerUs = 52e3, kPageableBytesPerUs = 10e3, kBothBytesPerUs = 72e3, kRowBytesPerUs = 3e6;
// One tile, us a channel (1024 and 4096 channels): row by row 0.18, packed rows of
// 16 bits 0.32 and of 32 bits 0.24; the plain kernel's small tiles 0.04 (at 2e12
// additions a second); shared sums 0.093 at 4 words per lane, 0.100 at 8, 0.183
// at 16.
double rows_tile_us(int nact, int nbits) { return nact * (nbits == 16 ? 0.32 : nbits == 32 ? 0.24 : 0.18); }
double plain_tile_us(int nact) { return 0.04 * nact; }
double pattern_tile_us(int nact, int lane_words) { return nact * (0.06 + 0.0075 * lane_words); }

double waves(size_t tiles, size_t sms) { return (double)((tiles + sms - 1) / sms); }

// DM groups of the last gulp, so that its device-to-host copy starts group by
// group. A group's launch takes whole waves of tiles; what shows is the first
// group and all copies, or all groups and the last copy.
size_t last_gulp_groups(const TddHostCall& h, size_t gc)
{
    const size_t blocks = (h.ndm + h.block_dms - 1) / h.block_dms;
    const size_t across = (gc + h.block_samples - 1) / h.block_samples;
    const double copy_us = (double)gc * (double)h.out_bytes / h.copy_rate;
    size_t best = 1;
    double least = 0;
    for (size_t n = 1; n <= std::min<size_t>(h.identity ? kMaxOutGroups : 1, blocks); ++n) {
        const double group = waves((blocks + n - 1) / n * across, h.sms) * h.tile_us + 10.0;
        const double us = std::max(group + copy_us, (double)n * group + copy_us / (double)n);
        if (n == 1 || us < least) {
            best = n;
            least = us;
        }
    }
    return best;
}

// The gulps (first output sample, samples) of a call in gulps of G. With host
// input and several gulps the first is a quarter of G: its input copy is the one
// that no kernel hides, and the next gulp's copy runs during its kernels.
std::vector<std::pair<size_t, size_t>> gulp_list(size_t nout, size_t G, size_t bt, bool host_in)
{
    std::vector<std::pair<size_t, size_t>> gulps;
    for (size_t g0 = 0; g0 < nout;) {
        size_t gc = std::min(G, nout - g0);
        if (g0 == 0 && host_in && gc < nout && G >= 4 * bt) gc = round_up(G / 4, bt);
        gulps.emplace_back(g0, gc);
        g0 += gc;
    }
    return gulps;
}

// Two input and two output buffers, one stream each for the copies in, the
// kernels and the copies out.
double host_call_us(const TddHostCall& h, size_t G)
{
    double in[2] = {0, 0}, kern[2] = {0, 0}, out[2] = {0, 0};  // ends of the last two gulps
    double in_bytes = 0;
    const auto gulps = gulp_list(h.nout, G, h.block_samples, true);
    const size_t blocks = (h.ndm + h.block_dms - 1) / h.block_dms;
    for (size_t i = 0; i < gulps.size(); ++i) {
        const size_t gc = gulps[i].second, a = i & 1;  // a: two gulps ago, then this one
        const double bytes = (double)(gc + h.tmax) * (double)h.row_bytes;
        in_bytes += bytes;
        in[a] = std::max(in[a ^ 1], kern[a]) + bytes / h.copy_rate + 8.0;
        double k = std::max({in[a], kern[a ^ 1], out[a]}) + (double)(gc + h.tmax) * (double)(4 * h.nchans + h.row_bytes) / kRowBytesPerUs;
        double o = out[a ^ 1];
        const size_t n = i + 1 == gulps.size() ? last_gulp_groups(h, gc) : 1;
        const size_t across = (gc + h.block_samples - 1) / h.block_samples;
        for (size_t g = 0; g < n; ++g) {
            k += waves((blocks + n - 1) / n * across, h.sms) * h.tile_us + 10.0;
            o = std::max(o, k) + (double)gc * (double)h.out_bytes / h.copy_rate / (double)n;
        }
        kern[a] = k;
        out[a] = o;
    }
    const double both = (in_bytes + (double)h.nout * (double)h.out_bytes) / kBothBytesPerUs;
    return std::max({out[0], out[1], both});
}
}  // namespace

TddEngine::TddEngine(GpuState& gpu) : m_gpu(gpu), m_setup(new Setup()) {}
TddEngine::~TddEngine()
{
    if (m_gpu.has_device) {
        rt::DeviceGuard g(m_gpu.device);
        cudaStreamSynchronize(m_gpu.stream());
        if (m_gpu.d2h) cudaStreamSynchronize(m_gpu.d2h->get());
        if (m_gpu.h2d) cudaStreamSynchronize(m_gpu.h2d->get());
    }
}

rt::Event& TddEngine::event(size_t i)
{
    while (m_events.size() <= i) m_events.emplace_back(new rt::Event(false));
    return *m_events[i];
}

void TddEngine::prepare(const TddView& v, const TddCall& c)
{
    Setup& s = *m_setup;
    // variants are numbered per input width; one outside the width's range
    // (or -1) selects the width's default, which is the pattern kernel where
    // that is the faster one
    const int eff_variant = (variant >= 0 && variant < kern::tiled_variant_count(c.in_nbits))
                                ? variant
                                : kern::tiled_default_variant(c.in_nbits);
    if (s.version == v.version && s.first == c.first_dm && s.count == c.dm_count &&
        s.nbits == c.in_nbits && s.kernel == kernel && s.variant == eff_variant) {
        choose_form(v, c);
        return;
    }

    s.version = ~0ul;  // the tables below are rewritten
    Setup n;
    n.version = v.version;
    n.first = c.first_dm;
    n.count = c.dm_count;
    n.nbits = c.in_nbits;
    n.kernel = kernel;
    n.variant = eff_variant;

    // Active channels (killmask != 0) and their multipliers. The reference
    // multiplies every sample by its killmask value (dedisperse_kernel.cuh:
    // 177-179); 0/1 masks let the tiled kernel skip channels and multiplies.
    bool general = false;
    for (size_t ch = 0; ch < v.nchans; ++ch) {
        const int32_t km = v.killmask[ch];
        if (km == 0) continue;
        if (km != 1) general = true;
        n.chan_list.push_back((int32_t)ch);
        n.km_vals.push_back((uint32_t)km);
    }
    n.nact = (int)n.chan_list.size();

    // DM range in ascending order (NaN sorts first: its delay is 0).
    const float* src = v.dms + c.first_dm;
    std::vector<int32_t> order(c.dm_count);
    std::iota(order.begin(), order.end(), 0);
    auto key = [&](int32_t i) {
        const float d = src[i];
        return std::isnan(d) ? -INFINITY : d;
    };
    n.identity = std::is_sorted(order.begin(), order.end(),
                                [&](int32_t a, int32_t b) { return key(a) < key(b); });
    if (!n.identity)
        std::stable_sort(order.begin(), order.end(),
                         [&](int32_t a, int32_t b) { return key(a) < key(b); });
    n.dms.resize(c.dm_count);
    for (size_t i = 0; i < c.dm_count; ++i) n.dms[i] = src[order[i]];
    if (!n.identity) n.perm = order;

    // Largest delay: d(dm, c) is monotonic in dm, so the extreme DMs bound it.
    const float dlo = n.dms.front(), dhi = n.dms.back();
    for (int j = 0; j < n.nact; ++j) {
        const float dl = v.delays[n.chan_list[j]];
        n.tmax = std::max(n.tmax, std::max(hostmath::delay_rn(dlo, dl), hostmath::delay_rn(dhi, dl)));
    }

    n.tiled_ok = (kernel != TddKernel::Plain) && !general;
    cudaStream_t st = m_gpu.stream();
    std::vector<int32_t> chan(n.chan_list);
    if (chan.empty()) chan.push_back((int32_t)v.nchans);
    // delay of each list entry (the padding channel's is 0)
    std::vector<float> cdl(chan.size());
    for (size_t j = 0; j < chan.size(); ++j) cdl[j] = chan[j] < (int32_t)v.nchans ? v.delays[chan[j]] : 0.f;
    n.pattern_ok = n.tiled_ok && n.variant == kern::tiled_default_variant(c.in_nbits) && n.nact &&
                   pattern_takes(n.dms, cdl, c.in_nbits);
    m_dms.reserve(n.dms.size() * 4);
    RT_CHECK(cudaMemcpyAsync(m_dms.get(), n.dms.data(), n.dms.size() * 4, cudaMemcpyHostToDevice, st));
    // (room for the padding that size_rows adds)
    m_chan.reserve((chan.size() + 256) * 4);
    RT_CHECK(cudaMemcpyAsync(m_chan.get(), chan.data(), chan.size() * 4, cudaMemcpyHostToDevice, st));
    m_cdl.reserve((cdl.size() + 256) * 4);
    RT_CHECK(cudaMemcpyAsync(m_cdl.get(), cdl.data(), cdl.size() * 4, cudaMemcpyHostToDevice, st));
    std::vector<uint32_t> km(n.km_vals);
    if (km.empty()) km.push_back(0);
    m_km.reserve(km.size() * 4);
    RT_CHECK(cudaMemcpyAsync(m_km.get(), km.data(), km.size() * 4, cudaMemcpyHostToDevice, st));
    if (!n.identity) {
        m_perm.reserve(n.perm.size() * 4);
        RT_CHECK(cudaMemcpyAsync(m_perm.get(), n.perm.data(), n.perm.size() * 4,
                                 cudaMemcpyHostToDevice, st));
    }
    // The host vectors must outlive the asynchronous copies.
    RT_CHECK(cudaStreamSynchronize(st));
    *m_setup = std::move(n);
    choose_form(v, c);
}

// The form that this call takes (after prepare): the pattern kernel with the
// period that suits the call's size where it is the faster one, else the
// row-by-row kernel of the chosen variant, else the plain one.
void TddEngine::choose_form(const TddView& v, const TddCall& c)
{
    Setup& s = *m_setup;
    if (keep_form && s.form_chosen) {
        choose_gulp(v, c, s.pattern);
        return;
    }
    s.pattern = false;
    const bool first_call = !s.form_chosen;
    s.tables_due = false;
    // an explicitly tiled plan is refused where the row-by-row form is
    if (kernel == TddKernel::Tiled) size_rows(v, c.in_nbits);
    if (kernel == TddKernel::Tiled && !s.rows_tiled)
        DD_THROW_MSG(DEDISP_UNKNOWN_ERROR, "tiled kernel unavailable for this killmask/DM list");
    if (s.pattern_ok && use_tables) {
        choose_gulp(v, c, true);
        const size_t nout = s.gulp;
        const size_t bt = (size_t)kern::pattern_block_samples(c.in_nbits, 4);
        const size_t tiles = (s.dms.size() + kern::kPatternDms - 1) / kern::kPatternDms * ((nout + bt - 1) / bt);
        cudaStream_t st = m_gpu.stream();
        auto later = [&] {
            if (first_call && !keep_form &&
                (double)s.dms.size() * s.nact * (double)(c.nsamps - v.max_delay) < kTablesAtOnce)
                return true;
            // tables take an allocation and a wait, which a capture must not see
            cudaStreamCaptureStatus cap = cudaStreamCaptureStatusNone;
            RT_CHECK(cudaStreamIsCapturing(st, &cap));
            return cap != cudaStreamCaptureStatusNone;
        };
        int J = kern::pattern_lane_words(c.in_nbits, tiles, s.group_words), i = 0;
        for (; J; J = kern::pattern_lane_words(c.in_nbits, tiles, s.group_words)) {
            i = table_index(J);
            if (s.table[i]) break;
            s.tables_due = later();
            if (s.tables_due) break;
            PatternTables& t = m_tables[i];
            bool use = t.size(m_dms.get<float>(), s.dms.size(), m_chan.get<int32_t>(), m_cdl.get<float>(),
                              (size_t)s.nact, v.nchans, c.in_nbits, J, st);
            if (use) {
                const PatternTables::Fit fit = t.fit(st);
                s.group_words = t.group_words();
                if (fit == PatternTables::kTooWide) continue;  // a shorter period, if one fits
                use = fit == PatternTables::kUse && t.emit(st);
            }
            s.table[i] = use ? 1 : -1;
            break;
        }
        s.pattern = J && s.table[i] == 1;
        s.lane_words = J;
    }
    // a list or mask that takes the row-by-row form keeps no tables
    if (!s.pattern && !s.tables_due && s.table[0] != 1 && s.table[1] != 1 && s.table[2] != 1) drop_idle_tables();
    if (!s.pattern) size_rows(v, c.in_nbits);
    s.tiled = s.pattern || s.rows_tiled;
    s.quad = s.pattern || s.rows_quad;
    s.period = s.pattern ? 32 * s.lane_words : s.rows_period;
    s.form_chosen = true;
    if (!s.pattern) choose_gulp(v, c, false);
}

// Output samples per pass: the user's cap, else the default, and for pinned host
// buffers, whose copies overlap the kernels, the gulps that take the least time
// in the model above (of the shared sums, or of the other forms) where that is at
// least 2% less than one gulp's. Pageable copies wait in the driver: no gain.
// Measured, ms, in one gulp; in eight or fewer of at least four times the overlap,
// whatever the trials and tiles; here: 1024 channels x 512 trials x 50000 samples
// 3.31, 4.03, 2.47; 1024 x 8 x 50000 (the input copy binds) 1.33, 1.92, 1.34;
// 4096 x 200 x 100000 12.4, 14.4, 10.5; 4096 x 16 x 20000 (each gulp a wave of
// 0.7 ms tiles) 3.0, 3.5, 2.4.
void TddEngine::choose_gulp(const TddView& v, const TddCall& c, bool shared)
{
    Setup& s = *m_setup;
    const bool host = !(c.flags & DEDISP_DEVICE_POINTERS), set = gulp_set && gulp_size;
    const size_t nout = c.nsamps - v.max_delay;
    s.gulp = std::min(nout, set ? gulp_size : host ? kHostDefaultGulp : kDefaultGulp);
    if (!host || set || !m_pinned) return;
    double least = 0.98 * host_call_us(host_call(v, c, shared, s.gulp), s.gulp);
    const size_t one = s.gulp;
    for (size_t k : {2, 3, 4, 6, 8, 12}) {
        size_t G = (nout + k - 1) / k;
        if (G >= one) continue;
        const TddHostCall h = host_call(v, c, shared, G);
        if (G > h.block_samples) G = G / h.block_samples * h.block_samples;
        const double us = host_call_us(h, G);
        if (us < least) {
            least = us;
            s.gulp = G;
        }
    }
}

// The model's numbers for a call in gulps of `gulp`, with the period that they
// would get.
TddHostCall TddEngine::host_call(const TddView& v, const TddCall& c, bool shared, size_t gulp) const
{
    const Setup& s = *m_setup;
    TddHostCall h{};
    h.nout = c.nsamps - v.max_delay;
    h.ndm = s.dms.size();
    h.tmax = s.tmax;
    h.row_bytes = v.nchans * (size_t)c.in_nbits / 8;
    h.out_bytes = h.ndm * (size_t)c.out_nbits / 8;
    h.nchans = v.nchans;
    h.identity = s.identity;
    h.sms = (size_t)kern::tdd_sm_count();
    h.copy_rate = m_pinned ? kPinnedBytesPerUs : kPageableBytesPerUs;
    if (shared) {
        h.block_dms = kern::kPatternDms;
        const size_t b = (size_t)kern::pattern_block_samples(c.in_nbits, 4);
        const size_t tiles = (h.ndm + h.block_dms - 1) / h.block_dms * ((gulp + b - 1) / b);
        const int J = std::max(4, kern::pattern_lane_words(c.in_nbits, tiles, s.group_words));
        h.block_samples = (size_t)kern::pattern_block_samples(c.in_nbits, J);
        h.tile_us = pattern_tile_us(s.nact, J);
    } else if (s.rows_tiled) {
        h.block_samples = (size_t)kern::tiled_block_samples(c.in_nbits, s.variant);
        h.block_dms = (size_t)kern::tiled_block_dms(c.in_nbits, s.variant);
        h.tile_us = rows_tile_us(s.nact, c.in_nbits);
    } else {
        h.block_samples = 16;
        h.block_dms = 32;
        h.tile_us = plain_tile_us(s.nact);
    }
    return h;
}

bool TddEngine::drop_idle_tables()
{
    Setup& s = *m_setup;
    bool any = false;
    for (int i = 0; i < 3; ++i) {
        if (s.pattern && i == table_index(s.lane_words)) continue;
        any = any || m_tables[i].held() > 0;
        m_tables[i].release();
        s.table[i] = std::min(s.table[i], 0);
    }
    return any;
}

// Window and stage sizes of the row-by-row tiled form, and its padded channel
// list.
void TddEngine::size_rows(const TddView& v, int nbits)
{
    Setup& s = *m_setup;
    if (s.rows_sized) return;
    s.rows_tiled = s.tiled_ok;
    if (s.rows_tiled) {
        const size_t ndm = s.dms.size();
        const int bd = kern::tiled_block_dms(nbits, s.variant);
        const int spw = 32 / nbits;
        const int J = kern::tiled_lane_words(nbits, s.variant);
        uint32_t span = 0;
        for (size_t t = 0; t < ndm; t += bd) {
            const float f = s.dms[t], l = s.dms[std::min(t + bd, ndm) - 1];
            for (int j = 0; j < s.nact; ++j) {
                const float dl = v.delays[s.chan_list[j]];
                const uint32_t a = hostmath::delay_rn(f, dl), b = hostmath::delay_rn(l, dl);
                span = std::max(span, a > b ? a - b : b - a);
            }
        }
        // quad-strided rows: a 1-sample delay is a 1-word offset, the window
        // is the lane set (P words) plus the span plus the 16-byte rounding
        s.rows_quad = kern::tiled_variant_quad(nbits, s.variant);
        s.rows_period = 32 * J;
        const size_t w = s.rows_quad ? (size_t)span + 3 + (size_t)s.rows_period
                                     : (span + 4 * (size_t)spw - 1) / spw + 32 * (size_t)J + 1;
        s.win_words = (int)round_up(w, 4);
        const int cs = w > ((size_t)1 << 26) ? 0 : kern::tiled_stage_channels(nbits, s.win_words, s.variant);
        if (cs < 2) {
            s.rows_tiled = s.rows_quad = false;
        } else {
            s.chan_per_stage = cs;
            s.nstages = std::max(1, (s.nact + cs - 1) / cs);
            std::vector<int32_t> chan(s.chan_list);
            chan.resize((size_t)s.nstages * s.chan_per_stage, (int32_t)v.nchans);
            std::vector<float> cdl(chan.size());
            for (size_t j = 0; j < chan.size(); ++j) cdl[j] = chan[j] < (int32_t)v.nchans ? v.delays[chan[j]] : 0.f;
            cudaStream_t st = m_gpu.stream();
            RT_CHECK(cudaStreamSynchronize(st));  // earlier calls read the shorter list
            m_chan.reserve(chan.size() * 4);
            m_cdl.reserve(cdl.size() * 4);
            RT_CHECK(cudaMemcpyAsync(m_chan.get(), chan.data(), chan.size() * 4, cudaMemcpyHostToDevice, st));
            RT_CHECK(cudaMemcpyAsync(m_cdl.get(), cdl.data(), cdl.size() * 4, cudaMemcpyHostToDevice, st));
            RT_CHECK(cudaStreamSynchronize(st));
        }
    }
    s.rows_sized = true;
}

void TddEngine::execute(const TddView& v, const TddCall& c)
{
    m_gpu.require_device();
    rt::DeviceGuard guard(m_gpu.device);
    stats = TddStats();

    const size_t nsamp_out = c.nsamps - v.max_delay;
    if (nsamp_out == 0 || c.dm_count == 0) return;
    m_pinned = !(c.flags & DEDISP_DEVICE_POINTERS) && rt::is_pinned_host(c.in) && rt::is_pinned_host(c.out);
    prepare(v, c);
    const Setup& s = *m_setup;
    stats.tiled = s.tiled;
    stats.form = s.pattern ? 2 : s.tiled ? 1 : 0;
    if (s.pattern) {
        stats.lane_words = s.lane_words;
        stats.rounds = m_tables[table_index(s.lane_words)].rounds();
    }

    const bool dev_in = (c.flags & DEDISP_DEVICE_POINTERS) != 0;
    const bool dev_out = dev_in;
    const int nbits = c.in_nbits;
    const size_t spw = 32 / nbits;
    const size_t ob = (size_t)c.out_nbits / 8;
    const size_t row_bytes = v.nchans * nbits / 8;
    const size_t ndm = c.dm_count;
    if (dev_out && c.out_stride % ob != 0)
        DD_THROW_MSG(DEDISP_INVALID_STRIDE, "device output stride must be a multiple of the sample size");

    const size_t bt = s.pattern ? (size_t)kern::pattern_block_samples(nbits, s.lane_words)
                      : s.tiled ? (size_t)kern::tiled_block_samples(nbits, s.variant)
                                : 16;
    const size_t win = s.tiled && !s.pattern ? (size_t)s.win_words : 0;

    // Gulp size: as chosen with the form, the grid limit, then device memory. With
    // more than one gulp the input rows and the output rows of a gulp have two
    // buffers each, so that gulp g+1's host-to-device copy and gulp g-1's
    // device-to-host copy run while gulp g is dedispersed.
    size_t G = s.gulp;
    G = std::min(G, (size_t)65535 * bt);
    if (G < nsamp_out && G > bt) G = G / bt * bt;  // whole time tiles in every gulp but the last
    auto pitch_for = [&](size_t g) {
        return round_up((round_up(g, bt) + s.tmax + spw - 1) / spw + win + 8, 32);
    };
    // quad-strided rows: the tile windows read up to word
    // (tiles - 1) * bt + tmax + P + 2 of a row (a pattern's series may start
    // or end a few words past its trials' reads)
    const bool quad = s.tiled && s.quad;
    const size_t slack = s.pattern ? 32 : 4;
    auto qpitch_for = [&](size_t g) { return round_up(round_up(g, bt) + s.tmax + s.period + slack, 32); };
    auto nbuf_for = [&](size_t g) -> size_t { return nsamp_out > g ? 2 : 1; };
    auto in_bytes_for = [&](size_t g) { return round_up(g + s.tmax, 128) * row_bytes; };
    // quad-strided rows are built straight from the input rows (K1d); the
    // channel-major packed copy exists only for the other forms
    auto bytes_for = [&](size_t g) {
        size_t b = quad ? (v.nchans + 1) * qpitch_for(g) * 4 : (v.nchans + 1) * pitch_for(g) * 4;
        if (!dev_out) b += nbuf_for(g) * ndm * g * ob;
        if (!dev_in) b += nbuf_for(g) * in_bytes_for(g);
        return b;
    };
    // buffers of an earlier call that are large enough need no look at the
    // free memory (64 channels, 32 trials, 8126 samples from host memory: 0.21
    // ms with it and a second wait for the error word, 0.135 without)
    const size_t nb = nbuf_for(G);
    const bool held = (quad ? m_q.capacity() >= (v.nchans + 1) * qpitch_for(G) * 4
                            : m_tr.capacity() >= (v.nchans + 1) * pitch_for(G) * 4) &&
                      (dev_out || std::min(m_out[0].capacity(), m_out[nb - 1].capacity()) >= ndm * G * ob) &&
                      (dev_in || std::min(m_stage[0].capacity(), m_stage[nb - 1].capacity()) >= in_bytes_for(G));
    if (!held) {
        size_t free_b = 0, total_b = 0;
        RT_CHECK(cudaMemGetInfo(&free_b, &total_b));
        const size_t own = m_tr.capacity() + m_q.capacity() + m_out[0].capacity() + m_out[1].capacity() +
                           m_stage[0].capacity() + m_stage[1].capacity();
        // tables of other calls go before the gulp shrinks
        if (bytes_for(G) > (free_b + own) / 100 * 90 && drop_idle_tables())
            RT_CHECK(cudaMemGetInfo(&free_b, &total_b));
        const size_t avail = free_b + own;
        while (G > bt && bytes_for(G) > avail / 100 * 90) G = round_up(G / 2, bt);
        if (bytes_for(G) > avail) {
            if (!s.pattern) DD_THROW(DEDISP_MEM_ALLOC_FAILED);
            // the row-by-row form needs no tables, and half the rows at 16 bits
            for (PatternTables& t : m_tables) t.release();
            m_setup->pattern_ok = false;
            execute(v, c);
            return;
        }
    }

    const size_t nbuf = nbuf_for(G);
    const size_t pitch = pitch_for(G);
    if (!quad) m_tr.reserve((v.nchans + 1) * pitch * 4);
    const size_t qpitch = quad ? qpitch_for(G) : 0;
    if (quad) {
        // room for the shared sums' rows too where they are still to come: a
        // captured graph of this call keeps its buffer when they do
        size_t words = 0;
        if (s.tables_due)
            for (int J : {4, 8, 16}) {
                const size_t b = (size_t)kern::pattern_block_samples(nbits, J);
                words = std::max(words, round_up(round_up(G, b) + s.tmax + 32 * (size_t)J + 32, 32));
            }
        if (words <= qpitch || !m_q.reserve_optional((v.nchans + 1) * words * 4))
            m_q.reserve((v.nchans + 1) * qpitch * 4);
    }
    for (size_t b = 0; b < nbuf; ++b) {
        if (!dev_out) m_out[b].reserve(ndm * G * ob);
        if (!dev_in) m_stage[b].reserve(in_bytes_for(G));
    }

    cudaStream_t ex = m_gpu.stream();
    cudaStream_t h2d = m_gpu.h2d->get();
    cudaStream_t d2h = m_gpu.d2h->get();
    uint32_t* tr = m_tr.get<uint32_t>();
    if (quad) {
        m_err.reserve(sizeof(unsigned));
        RT_CHECK(cudaMemsetAsync(m_err.get(), 0, sizeof(unsigned), ex));
    }

    const float in_range = (float)(nbits == 32 ? 0xFFFFFFFFu : ((1u << nbits) - 1u));
    const float den = in_range * (float)v.nchans;
    const float factor = 3.f * 1024.f / 255.f / 16.f;

    // The last gulp's K2 runs per group of DM slots whose output rows are
    // contiguous, so that its device-to-host copy starts group by group
    // (every other gulp's copy already overlaps the next gulp's kernels, and
    // each extra launch ends with a partly filled wave: last_gulp_groups).
    const size_t bd = s.tiled && !s.pattern ? (size_t)kern::tiled_block_dms(nbits, s.variant) : 32;
    const size_t ntile = (ndm + bd - 1) / bd;
    size_t ngroups_last = (!dev_out && s.identity) ? std::min<size_t>(kMaxOutGroups, ntile) : 1;

    const std::vector<std::pair<size_t, size_t>> gulps = gulp_list(nsamp_out, G, bt, !dev_in);
    if (ngroups_last > 1)
        ngroups_last = last_gulp_groups(host_call(v, c, s.pattern, G), gulps.back().second);

    std::unique_ptr<rt::Event> t_a, t_b, t_c;
    if (record_timing) {
        t_a.reset(new rt::Event(true));
        t_b.reset(new rt::Event(true));
        t_c.reset(new rt::Event(true));
    }

    size_t ev = 0;
    rt::Event* ev_in_free[2] = {&event(ev++), &event(ev++)};   // K1 has read input buffer b
    rt::Event* ev_out_free[2] = {&event(ev++), &event(ev++)};  // D2H has read output buffer b
    bool in_used[2] = {false, false}, out_used[2] = {false, false};

    for (size_t gi = 0; gi < gulps.size(); ++gi) {
        const size_t g0 = gulps[gi].first, gc = gulps[gi].second;
        const bool last = gi + 1 == gulps.size();
        const size_t ngroups = last ? ngroups_last : 1;
        const size_t b = gi % nbuf;
        const size_t rows_need = gc + s.tmax;
        const size_t rows_avail = std::min(rows_need, c.nsamps - g0);

        if (t_a && g0 == 0) t_a->record(ex);
        // Padding channel row (all zero).
        if (quad) RT_CHECK(cudaMemsetAsync(m_q.get<uint32_t>() + v.nchans * qpitch, 0, qpitch * 4, ex));
        else RT_CHECK(cudaMemsetAsync(tr + v.nchans * pitch, 0, pitch * 4, ex));

        // K1 (channel-major packed) or K1d (quad-strided rows) from the
        // gulp's input rows, zero past the data.
        const uint8_t* rows = c.in + g0 * c.in_stride;
        size_t rows_pitch = c.in_stride;
        if (!dev_in) {
            // the whole gulp's rows into input buffer b, on the copy stream
            if (in_used[b]) RT_CHECK(cudaStreamWaitEvent(h2d, *ev_in_free[b], 0));
            RT_CHECK(cudaMemcpy2DAsync(m_stage[b].get(), row_bytes, rows, c.in_stride, row_bytes, rows_avail,
                                       cudaMemcpyHostToDevice, h2d));
            rt::Event& ready = event(ev++);
            ready.record(h2d);
            RT_CHECK(cudaStreamWaitEvent(ex, ready, 0));
            rows = m_stage[b].get<uint8_t>();
            rows_pitch = row_bytes;
        }
        if (quad) {
            kern::QuadDirectArgs qa{rows, rows_pitch, rows_avail, v.nchans, nbits, m_q.get<uint32_t>(), qpitch,
                                    s.period};
            kern::launch_quad_direct(qa, ex);
        } else {
            kern::TransposeArgs ta{rows, rows_pitch, rows_avail, v.nchans, nbits, tr, pitch, 0, pitch};
            kern::launch_transpose(ta, ex);
        }
        ++stats.launches;
        if (!dev_in) {
            ev_in_free[b]->record(ex);
            in_used[b] = true;
        }
        if (t_b && g0 == 0) t_b->record(ex);

        // K2 per DM group.
        if (!dev_out && out_used[b]) RT_CHECK(cudaStreamWaitEvent(ex, *ev_out_free[b], 0));
        const size_t out_elems_stride = dev_out ? c.out_stride / ob : gc;
        uint8_t* out_base = dev_out ? c.out + g0 * ob : m_out[b].get<uint8_t>();
        std::vector<std::pair<size_t, size_t>> groups;
        for (size_t gr = 0; gr < ngroups; ++gr) {
            const size_t t0 = ntile * gr / ngroups, t1 = ntile * (gr + 1) / ngroups;
            const size_t s0 = t0 * bd, s1 = std::min(ndm, t1 * bd);
            if (s0 >= s1) continue;
            groups.emplace_back(s0, s1);
            kern::DedisperseArgs da{};
            da.tr = quad ? m_q.get<uint32_t>() : tr;
            da.tr_pitch_words = quad ? qpitch : pitch;
            da.nbits = nbits;
            da.nchans = v.nchans;
            da.chan_list = m_chan.get<int32_t>();
            da.nact = s.nact;
            da.nstages = s.nstages;
            da.km_vals = m_km.get<uint32_t>();
            da.delay_table = m_gpu.delay_table.get<float>();
            da.chan_delay = m_cdl.get<float>();
            da.dms = m_dms.get<float>() + s0;
            da.ndm = (int)(s1 - s0);
            da.nsamp_out = gc;
            da.out_stride = out_elems_stride;
            da.out_nbits = c.out_nbits;
            da.den = den;
            da.factor = factor;
            da.win_words = s.win_words;
            da.chan_per_stage = s.chan_per_stage;
            da.variant = s.variant;
            da.err = m_err.get<unsigned>();
            if (s.identity) {
                da.perm = nullptr;
                da.out = out_base + s0 * out_elems_stride * ob;
            } else {
                da.perm = m_perm.get<int32_t>() + s0;
                da.out = out_base;
            }
            if (s.pattern) {
                m_tables[table_index(s.lane_words)].fill(da, s0 / bd);  // s0 is a multiple of bd
                kern::launch_dedisperse_pattern(da, ex);
            } else if (s.tiled) kern::launch_dedisperse_tiled(da, ex);
            else kern::launch_dedisperse_plain(da, ex);
            ++stats.launches;
            if (!dev_out) event(ev + groups.size() - 1).record(ex);
        }
        if (t_c && last) t_c->record(ex);

        // D2H per group into the caller's rows (column offset g0).
        if (!dev_out) {
            for (size_t gr = 0; gr < groups.size(); ++gr) {
                const size_t s0 = groups[gr].first, s1 = groups[gr].second;
                const size_t r0 = s.identity ? s0 : 0, nrow = s.identity ? s1 - s0 : ndm;
                RT_CHECK(cudaStreamWaitEvent(d2h, event(ev + gr), 0));
                if (!s.identity && gr + 1 < groups.size()) continue;
                RT_CHECK(cudaMemcpy2DAsync(c.out + r0 * c.out_stride + g0 * ob, c.out_stride,
                                           m_out[b].get<uint8_t>() + r0 * gc * ob, gc * ob, gc * ob,
                                           nrow, cudaMemcpyDeviceToHost, d2h));
            }
            ev += groups.size();
            ev_out_free[b]->record(d2h);
            out_used[b] = true;
        }
    }

    const bool async = (c.flags & DEDISP_ASYNC) && dev_in;
    if (!async) {
        // the error word comes back behind the kernels, before the one wait (a
        // copy to pageable memory, should there be no pinned word, waits itself
        // and takes 2 us more: 44.5 against 46.8 for 64 channels x 32 trials x
        // 2048 samples)
        unsigned pageable = 0;
        unsigned* failed = quad ? m_err_host.get() : nullptr;
        if (!failed) failed = &pageable;
        if (quad) RT_CHECK(cudaMemcpyAsync(failed, m_err.get(), sizeof(unsigned), cudaMemcpyDeviceToHost, ex));
        RT_CHECK(cudaStreamSynchronize(ex));
        if (!dev_out) RT_CHECK(cudaStreamSynchronize(d2h));
        if (*failed)
            DD_THROW_MSG(DEDISP_INTERNAL_GPU_ERROR, "a staged window copy did not complete");
    }
    if (record_timing) {
        RT_CHECK(cudaEventSynchronize(*t_c));
        RT_CHECK(cudaEventElapsedTime(&stats.transpose_ms, *t_a, *t_b));
        RT_CHECK(cudaEventElapsedTime(&stats.kernel_ms, *t_b, *t_c));
    }
}

}  // namespace detail
}  // namespace dedisp
