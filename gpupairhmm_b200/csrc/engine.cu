// Host-side engine: batch validation and indexing, device buffers and the
// per-batch launch sequence.
//
// Launch sequence of one batch:
//   pack                        caller SoA -> packed HBM layout; the batch's fills
//   bin_count, hist_scan,
//   bin_scatter                 sorted work list
//   fp32_tile_kernel,
//   fp32_bucket_kernel          one launch per non-empty length bucket: exact tiles for reads
//                               of 33-4,096 positions, else (user tables, the plain form, engines
//                               without the FP64 pass) padded ones
//   fp64_tile_kernel,
//   fp64_rescue_kernel          per length class, pairs flagged by the FP32 pass in doubles,
//                               then the few beyond the scaled doubles' range
// A stage's launches fork onto side streams and join back.  Small batches that repeat are
// launched as one graph (run_pipeline).
// Compared with the reference executor (gpuworker.cuh:559-973) there is no
// device-to-host synchronisation inside a batch: the host derives bucket sizes
// and every bucket's range of work items from the record structure it already
// holds.
#include <algorithm>
#include <bitset>
#include <chrono>
#include <cmath>
#include <cstring>
#include <memory>
#include <thread>

#include "engine.hpp"

namespace phmm {

namespace {

constexpr int64_t kScratchBudget = int64_t(4) << 30;  // border scratch cap per batch

// Device counters of a batch (one array, zeroed by the fill kernel): bucket
// task counters, then per FP64 length class the scaled tier's list counts, the
// extended tier's list counts, and the two tiers' task counters.
constexpr int kCtrScaled = kMaxBuckets;
constexpr int kCtrExt = kMaxBuckets + kMaxFp64Classes;
constexpr int kCtrTaskScaled = kMaxBuckets + 2 * kMaxFp64Classes;
constexpr int kCtrTaskExt = kMaxBuckets + 3 * kMaxFp64Classes;
constexpr int kCtrTotal = kMaxBuckets + 4 * kMaxFp64Classes;
// FP64 groups, in warps, up to which the lists are not sorted by haplotype length: at most
// a few rounds of resident warps, so the order decides little and the three launches of
// the sort are a third of the stage of a small batch.  Unsorted / sorted: one uneven region
// 175 / 189 us, one long-read region (64 pairs on 8 warps each) 2.49 / 2.52 ms, 64 long-read
// regions (4,096 pairs on 4 warps each) 21.3 / 20.5 ms.
constexpr int64_t kNoSortWarps = 4096;
// Batches of more pairs or length classes than this, or whose launches have not been the
// same for a while, are launched kernel by kernel (see run_pipeline).
constexpr int64_t kGraphMaxPairs = 4096;
constexpr int kGraphMaxClasses = 6;
constexpr int64_t kGraphAfter = 8;
// multi-tile FP64 pairs up to which the two tiers run fused (about one round of
// resident warps of that class's kernel on 148 SMs)
constexpr int64_t kFuseMaxPairs = 2048;

// Reads beyond this count as multi-tile (the stats' multi_tile_pairs, the serving
// queue's slots), on whatever kernel they run.
constexpr int kLongRead = 1024;

// Exact tiles for reads of lo+1 .. hi positions on groups of G lanes, one rule per
// R (a lane's positions).
void add_exact_rules(std::vector<TileRule>& rules, int G, int lo, int hi) {
    for (int R = lo / G + 1; R * G <= hi; ++R)
        rules.push_back({R * G, G, R, R * G > kLongRead, G <= 32, true});
}

std::vector<TileRule> engine_default_rules() {
    // The two shortest classes keep the padded tiles autotune.py picked for them;
    // from 33 positions on exact tiles with as many positions per lane as fit (the
    // per-step work of a lane is amortised over them) and at least 11 once a group
    // of 16 or 32 lanes is needed.  Reads of 641-2,048 positions: one warp with two or
    // three parts in turn; beyond, blocks of 8 warps.
    std::vector<TileRule> rules = {{16, 4, 4, false, false}, {32, 4, 8, false, true}};
    add_exact_rules(rules, 8, 32, 160);
    add_exact_rules(rules, 16, 160, 320);
    add_exact_rules(rules, 32, 320, 640);
    add_exact_rules(rules, 64, 640, 1536);
    add_exact_rules(rules, 96, 1536, 2016);
    add_exact_rules(rules, 256, 1792, 4096);
    rules.push_back({1 << 30, 32, 32, true});
    return rules;
}

std::vector<TileRule> plain_rules() {
    // The reference's generic single-tile table (tuningconfigs.hpp:33-57) and
    // its multi-tile configuration for longer reads (gpuworker.cuh:189-194).
    return {
        {16, 4, 4, false},     {32, 4, 8, false},     {48, 4, 12, false},    {64, 4, 16, false},
        {80, 4, 20, false},    {96, 4, 24, false},    {112, 4, 28, false},   {128, 4, 32, false},
        {160, 8, 20, false},   {192, 8, 24, false},   {224, 8, 28, false},   {256, 8, 32, false},
        {320, 16, 20, false},  {384, 16, 24, false},  {448, 16, 28, false},  {512, 16, 32, false},
        {640, 32, 20, false},  {768, 32, 24, false},  {896, 32, 28, false},  {1024, 32, 32, false},
        {1 << 30, 32, 16, true},
    };
}

std::vector<TileRule> gcp_rules() {
    // gcp mode (eps and beta per read): the exact tiles, and around them the padded
    // scalar kernels compiled with that option (fp32_gcp.cu).
    std::vector<TileRule> rules = {{32, 4, 16, false}};
    add_exact_rules(rules, 8, 32, 160);
    add_exact_rules(rules, 16, 160, 320);
    add_exact_rules(rules, 32, 320, 640);
    add_exact_rules(rules, 64, 640, 1536);
    add_exact_rules(rules, 96, 1536, 2016);
    add_exact_rules(rules, 256, 1792, 4096);
    rules.push_back({1 << 30, 32, 32, true});
    return rules;
}

// Tables of an engine without the FP64 pass: padded tiles (autotune.py's picks; in gcp
// mode the kernels compiled with that option).  A score then is what single precision
// gives, down to the end of its range, and values on exact tiles lie up to 1/delta lower:
// between 1e-72 and 1e-76 scores of reads with gap qualities 60-93 were off by 0.07 (rms
// of log10) or -inf there, and are good to 2e-6 on these.
std::vector<TileRule> padded_rules(bool gcp) {
    if (gcp)
        return {
            {64, 4, 16, false},   {128, 8, 16, false},   {160, 8, 20, false},    {256, 16, 16, false},
            {512, 32, 16, false}, {1024, 32, 32, false}, {1 << 30, 32, 32, true},
        };
    return {
        {16, 4, 4, false},         {32, 4, 8, false, true},    {48, 4, 12, false, true},  {64, 4, 16, false},
        {80, 4, 20, false},        {96, 8, 12, false, true},   {112, 4, 28, false},       {128, 8, 16, false, true},
        {144, 8, 18, false},       {160, 8, 20, false},        {176, 8, 22, false},       {192, 16, 12, false, true},
        {224, 8, 28, false},       {256, 16, 16, false, true}, {288, 16, 18, false},      {320, 16, 20, false},
        {384, 32, 12, false, true}, {448, 16, 28, false},      {512, 32, 16, false, true}, {640, 32, 20, false},
        {768, 32, 24, false},      {896, 32, 28, false},       {1024, 32, 32, false},     {1280, 32, 20, true},
        {1536, 32, 24, true},      {1792, 32, 28, true},       {1 << 30, 32, 32, true},
    };
}

// The table of a batch of few pairs: the same, with 32 lanes a group wherever an
// exact tile has fewer, and blocks of 8 warps (256 lanes) from 641 positions on.  Results do not change: the exact tiles' do not depend on the
// shape, and the other classes stay.
std::vector<TileRule> small_rules(const std::vector<TileRule>& rules) {
    std::vector<TileRule> small;
    for (size_t i = 0; i < rules.size(); ++i) {
        if (!rules[i].exact || rules[i].G == 256) {
            small.push_back(rules[i]);
            continue;
        }
        if (rules[i].G > 32) {   // 641-2,016 positions; the blocks start at 1,793
            while (i + 1 < rules.size() && rules[i + 1].exact && rules[i + 1].G < 256) ++i;
            add_exact_rules(small, 256, 512, 1792);
            continue;
        }
        const int lo = i ? rules[i - 1].max_len : 0;
        while (i + 1 < rules.size() && rules[i + 1].exact && rules[i + 1].G <= 32) ++i;
        add_exact_rules(small, 32, lo, rules[i].max_len);
    }
    return small;
}

// FP64 classes: exact tiles on groups of 8-32 lanes (wide: 32); from 641 positions on
// blocks of 4 warps (wide, and from 2,049 on: 8); padded kernels for the shortest and
// the longest reads.  One warp with the parts in turn was no faster where the pairs
// fill the chip (400 long-read regions 74.5 against 75.1 ms, 64 regions 13.8 against
// 13.3), although it can stop at a part's end, and needs border rows in memory.  The
// extended tier, which few pairs reach, has the padded kernels up to 640 positions.
pairhmm_status_t make_fp64_table(bool wide, bool gcp, Fp64Table& t) {
    struct Span { int G, lo, hi; };
    const std::vector<Span> narrow = {{8, 32, 160}, {16, 160, 320}, {32, 320, 640}};
    std::vector<Span> spans = wide ? std::vector<Span>{{32, 32, 640}} : narrow;
    if (wide) spans.push_back({256, 512, 2048});   // from 641 on: the classes before it end there
    else spans.push_back({128, 640, 2048});
    spans.push_back({256, 2048, 4096});
    struct Padded { int max_len, G, R; };
    static constexpr Padded kExt[] = {{64, 4, 16},   {96, 8, 12},    {128, 8, 16}, {160, 16, 10},
                                      {192, 16, 12}, {256, 16, 16}, {640, 32, 16}};
    auto ext_of = [&](int hi, int G, int R) {
        // padded extended kernels are shared by the classes within their bound
        if (G <= 32 && hi <= 640) {
            const Padded* e = kExt;
            while (hi > e->max_len) ++e;
            const Fp64Config* cfg = find_fp64_config(e->G, e->R, false, true, gcp);
            if (!t.exts.empty() && t.exts.back().cfg == cfg) return (int)t.exts.size() - 1;
            t.exts.push_back({cfg, 0, 0, false});
        } else {
            // blocks of 8 warps whatever the scaled tier has: few pairs come this far, and one
            // warp alone would still be on its first pair when the other classes are done
            t.exts.push_back({G > 32 ? find_fp64_config(256, (hi + 255) / 256, true, true, gcp)
                                     : find_fp64_config(G, R, false, true, gcp), 0, 0, true});
        }
        return (int)t.exts.size() - 1;
    };
    auto add = [&](int hi, int G, int R, bool exact) {
        t.classes.push_back({hi, find_fp64_config(G, R, exact, false, gcp), ext_of(hi, G, R)});
    };
    add(32, 4, 16, false);
    for (const Span& sp : spans)
        for (int R = sp.lo / sp.G + 1; R * sp.G <= sp.hi; ++R) add(R * sp.G, sp.G, R, true);
    add(INT32_MAX, 32, 16, false);
    t.fused = find_fp64_config(32, 16, false, false, gcp, true);
    if (!t.fused || t.classes.size() > kMaxFp64Classes) return PAIRHMM_ERR_UNSUPPORTED;
    for (size_t c = 0; c < t.classes.size(); ++c) {
        Fp64Table::Ext& e = t.exts[t.classes[c].ext];
        if (!t.classes[c].scaled || !e.cfg) return PAIRHMM_ERR_UNSUPPORTED;
        const Fp64Config& k = *t.classes[c].scaled;   // exact: more than G*(R-1) positions
        if (k.exact && (c ? t.classes[c - 1].max_len : 0) < k.G * (k.R - 1)) return PAIRHMM_ERR_UNSUPPORTED;
        if (c == 0 || t.classes[c - 1].ext != t.classes[c].ext) e.first = (int)c;
        e.last = (int)c;
    }
    t.lut.resize(kFp64LutSize);
    for (int L = 0, c = 0; L < kFp64LutSize; ++L) {
        while (L > t.classes[c].max_len) ++c;
        t.lut[L] = (uint8_t)c;
    }
    return PAIRHMM_OK;
}

inline int64_t round_up(int64_t x, int64_t m) { return (x + m - 1) / m * m; }

int bucket_of_host(int L, const std::vector<TileRule>& rules) {
    int b = 0;
    const int nb = (int)rules.size();
    while (b < nb - 1 && L > rules[b].max_len) ++b;
    return b;
}

}  // namespace

cudaError_t DevBuf::ensure(size_t bytes) {
    if (bytes <= cap && ptr) return cudaSuccess;
    release();
    size_t want = std::max<size_t>(bytes + bytes / 4, 256);
    cudaError_t e = pool ? cudaMallocFromPoolAsync(&ptr, want, pool, stream) : cudaMalloc(&ptr, want);
    if (e != cudaSuccess) {
        ptr = nullptr;
        cap = 0;
        return e;
    }
    cap = want;
    return cudaSuccess;
}

void DevBuf::release() {
    if (ptr) {
        if (pool) cudaFreeAsync(ptr, stream);
        else cudaFree(ptr);
    }
    ptr = nullptr;
    cap = 0;
}

namespace {
// what is wrong with a tile table (null: nothing)
const char* check_rules(const std::vector<TileRule>& rules, bool gcp) {
    if (rules.empty() || (int)rules.size() > kMaxBuckets) return "tile table size";
    for (size_t i = 0; i < rules.size(); ++i) {
        if (rules[i].packed && rules[i].multi_tile)
            return "packed rules are single tile";
        if (!find_fp32_config(rules[i].G, rules[i].R, rules[i].multi_tile, rules[i].packed, rules[i].exact,
                              gcp))
            return "tile table names a configuration that is not compiled";
        if (i > 0 && rules[i].max_len <= rules[i - 1].max_len)
            return "tile table bounds must increase";
        if ((!rules[i].multi_tile || rules[i].exact) && rules[i].max_len > rules[i].G * rules[i].R)
            return "single-tile rule shorter than its bucket";
        if (rules[i].exact && (i ? rules[i - 1].max_len : 0) < rules[i].G * (rules[i].R - 1))
            return "exact tile for reads of fewer positions than it takes";
    }
    if (!rules.back().multi_tile || rules.back().exact) return "last rule must be multi-tile";
    return nullptr;
}

std::vector<TileRule> default_rules(const pairhmm_options_t& o) {
    if (o.mode == PAIRHMM_MODE_PLAIN) return plain_rules();
    if (!o.fp64_rescue) return padded_rules(o.gcp != 0);
    return o.gcp ? gcp_rules() : engine_default_rules();
}
}  // namespace

Engine::Engine(const pairhmm_options_t& opts) : opts_(opts) { tables_[0].rules = default_rules(opts_); }

std::vector<DevBuf*> Engine::all_buffers() {
    return {&ph2pr_, &in_read_bases_, &in_bq_,
            &in_iq_, &in_dq_, &in_read_off_, &in_read_len_, &in_hap_bases_, &in_hap_off_, &in_hap_len_,
            &read_record_, &read_local_, &rec_haps_, &rec_hap_base_, &rec_pair_base_, &read_start_,
            &hap_start_, &read_pack_, &read_meta_, &hap_code_, &hist_, &cursor_, &items_, &rescue_, &counters_,
            &scores_, &scratch_, &unit_read0_, &unit_read1_, &unit_bucket_, &arena_, &rescue_off_,
            &rescue_ext_, &rsort_, &fp64_lut_[0], &fp64_lut_[1],
            &in_gq_, &read_gcp_};
}

Engine::~Engine() {
    if (ready_) cudaSetDevice(opts_.device);
    if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
    for (DevBuf* b : all_buffers()) b->release();
    if (stream_) cudaStreamSynchronize(stream_);
    if (pool_) cudaMemPoolDestroy(pool_);
    if (host_hdr_) cudaFreeHost(host_hdr_);
    if (ev0_) cudaEventDestroy(ev0_);
    if (ev1_) cudaEventDestroy(ev1_);
    if (ev_prep_) cudaEventDestroy(ev_prep_);
    if (ev_fp32_) cudaEventDestroy(ev_fp32_);
    for (int i = 0; i < kSideStreams; ++i) {
        if (join_[i]) cudaEventDestroy(join_[i]);
        if (side_[i]) cudaStreamDestroy(side_[i]);
    }
    if (fork_) cudaEventDestroy(fork_);
    if (span0_) cudaEventDestroy(span0_);
    if (span1_) cudaEventDestroy(span1_);
    if (stream_) cudaStreamDestroy(stream_);
}

pairhmm_status_t Engine::fail(pairhmm_status_t s, const std::string& msg) {
    last_error_ = msg;
    return s;
}

pairhmm_status_t Engine::cuda_fail(cudaError_t e, const char* what) {
    last_error_ = std::string(what) + ": " + cudaGetErrorString(e);
    return e == cudaErrorMemoryAllocation ? PAIRHMM_ERR_OUT_OF_MEMORY : PAIRHMM_ERR_CUDA;
}

#define PHMM_CUDA(call)                                   \
    do {                                                  \
        cudaError_t e_ = (call);                          \
        if (e_ != cudaSuccess) return cuda_fail(e_, #call); \
    } while (0)

pairhmm_status_t Engine::reserve_pool(size_t bytes) {
    if (!pool_ || bytes == 0) return PAIRHMM_OK;
    PHMM_CUDA(cudaSetDevice(opts_.device));
    void* p = nullptr;
    PHMM_CUDA(cudaMallocFromPoolAsync(&p, bytes, pool_, stream_));
    PHMM_CUDA(cudaFreeAsync(p, stream_));
    PHMM_CUDA(cudaStreamSynchronize(stream_));
    return PAIRHMM_OK;
}

pairhmm_status_t Engine::ensure_side_streams(int n) {
    for (int i = 0; i < n; ++i) {
        if (!side_[i]) PHMM_CUDA(cudaStreamCreateWithFlags(&side_[i], cudaStreamNonBlocking));
        if (!join_[i]) PHMM_CUDA(cudaEventCreateWithFlags(&join_[i], cudaEventDisableTiming));
    }
    return PAIRHMM_OK;
}

pairhmm_status_t Engine::init() {
    int ndev = 0;
    cudaError_t e = cudaGetDeviceCount(&ndev);
    if (e != cudaSuccess || ndev == 0) return fail(PAIRHMM_ERR_UNSUPPORTED, "no CUDA device");
    if (opts_.device < 0 || opts_.device >= ndev) return fail(PAIRHMM_ERR_INVALID_ARGUMENT, "bad device ordinal");
    if (opts_.gcp && opts_.mode == PAIRHMM_MODE_PLAIN)
        return fail(PAIRHMM_ERR_INVALID_ARGUMENT, "gcp mode runs in the engine form, not the plain form");
    PHMM_CUDA(cudaSetDevice(opts_.device));
    cudaDeviceProp prop{};
    PHMM_CUDA(cudaGetDeviceProperties(&prop, opts_.device));
    if (prop.major < 10) return fail(PAIRHMM_ERR_UNSUPPORTED, "the kernels are built for sm_100a");
    num_sms_ = prop.multiProcessorCount;
    PHMM_CUDA(cudaStreamCreateWithFlags(&stream_, cudaStreamNonBlocking));
    PHMM_CUDA(cudaEventCreateWithFlags(&fork_, cudaEventDisableTiming));
    {
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = opts_.device;
        PHMM_CUDA(cudaMemPoolCreate(&pool_, &props));
        uint64_t keep = UINT64_MAX;
        PHMM_CUDA(cudaMemPoolSetAttribute(pool_, cudaMemPoolAttrReleaseThreshold, &keep));
        for (DevBuf* b : all_buffers()) {
            b->pool = pool_;
            b->stream = stream_;
        }
    }
    PHMM_CUDA(cudaMallocHost(&host_hdr_, sizeof(unsigned long long) * 2 * kMaxFp64Classes));
    PHMM_CUDA(cudaEventCreate(&ev0_));
    PHMM_CUDA(cudaEventCreate(&ev1_));
    PHMM_CUDA(cudaEventCreate(&ev_prep_));
    PHMM_CUDA(cudaEventCreate(&ev_fp32_));

    // probability table p(q) = float(10^(-q/10)) (gpuworker.cuh:473-486)
    float table[128];
    for (int i = 0; i < 128; ++i) table[i] = (float)std::pow(10.0, (-i) / 10.0);
    PHMM_CUDA(ph2pr_.ensure(sizeof(table)));
    PHMM_CUDA(cudaMemcpy(ph2pr_.ptr, table, sizeof(table), cudaMemcpyHostToDevice));
    PHMM_CUDA(counters_.ensure(sizeof(unsigned long long) * kCtrTotal));
    // FP64 list sort: per-class histogram (uint32) then cursors (uint64)
    PHMM_CUDA(rsort_.ensure((sizeof(unsigned int) + sizeof(unsigned long long)) * kMaxFp64Classes * kRescueHBins));
    for (int w = 0; w < 2; ++w) {
        if (make_fp64_table(w == 1, opts_.gcp != 0, fp64_tables_[w]) != PAIRHMM_OK)
            return fail(PAIRHMM_ERR_UNSUPPORTED, "FP64 class without compiled kernel");
        PHMM_CUDA(fp64_lut_[w].ensure(kFp64LutSize));
        PHMM_CUDA(cudaMemcpy(fp64_lut_[w].ptr, fp64_tables_[w].lut.data(), kFp64LutSize, cudaMemcpyHostToDevice));
    }
    ready_ = true;
    return build_tables(default_rules(opts_));
}

pairhmm_status_t Engine::set_tile_table(const std::vector<TileRule>& rules) {
    if (twin_) {
        const pairhmm_status_t t = twin_->set_tile_table(rules);
        if (t != PAIRHMM_OK) return fail(t, twin_->last_error());
    }
    const char* wrong = check_rules(rules, opts_.gcp != 0);
    if (wrong) return fail(PAIRHMM_ERR_INVALID_ARGUMENT, wrong);
    if (graph_exec_) cudaGraphExecDestroy(graph_exec_);
    graph_exec_ = nullptr;
    last_shape_.clear();
    shape_repeats_ = 0;
    if (ready_) return build_tables(rules);
    tables_[0].rules = rules;
    return PAIRHMM_OK;
}

bool Engine::has_default_table(const std::vector<TileRule>& rules) const {
    return opts_.mode != PAIRHMM_MODE_PLAIN && rules == default_rules(opts_);
}

pairhmm_status_t Engine::build_tables(const std::vector<TileRule>& rules) {
    TileTable built[2];
    built[0].rules = rules;
    if (has_default_table(rules) && opts_.fp64_rescue) built[1].rules = small_rules(rules);
    for (TileTable& t : built) {
        const char* wrong = t.rules.empty() ? nullptr : check_rules(t.rules, opts_.gcp != 0);
        if (wrong) return fail(PAIRHMM_ERR_INVALID_ARGUMENT, wrong);
        for (const TileRule& r : t.rules) {
            t.cfg.push_back(find_fp32_config(r.G, r.R, r.multi_tile, r.packed, r.exact, opts_.gcp != 0));
            if (!t.cfg.back()) return fail(PAIRHMM_ERR_INVALID_ARGUMENT, "tile rule without compiled kernel");
        }
    }
    for (int i = 0; i < 2; ++i) tables_[i] = std::move(built[i]);
    table_ = &tables_[0];
    return PAIRHMM_OK;
}

// A batch of few pairs leaves most of the chip idle and takes as long as its longest
// pair, one step per haplotype position; on 32 lanes instead of 8 or 16 a step works
// on a quarter or half of the positions.  What counts is the pairs per length class:
// the classes are launches of their own, each with its own last wave.  FP32 stage,
// table for few / for many pairs: reads of one length (100) 128 pairs 0.018 / 0.029 ms,
// 2,048 pairs 0.027 / 0.029, 4,096 pairs 0.045 / 0.031; (250) 1,024 pairs 0.043 / 0.062,
// 2,048 pairs 0.072 / 0.066; uneven regions (13 classes) 395 pairs 0.057 / 0.088,
// 6,500 pairs 0.19 / 0.24, 13,000 pairs 0.31 / 0.29, 27,000 pairs 0.48 / 0.40.
// A long read's pair counts as the 8 warps it takes in the small table.
void Engine::choose_table(int64_t num_records, const int32_t* reads_per_record, const int32_t* haps_per_record,
                          const int32_t* read_lengths, int64_t pairs) {
    table_ = &tables_[0];
    fp64_ = &fp64_tables_[0];
    if (tables_[1].rules.empty() || pairs > kSmallPairs * (int64_t)tables_[0].rules.size()) return;
    std::bitset<kMaxBuckets> seen;
    int64_t weight = 0, i = 0;
    for (int64_t g = 0; g < num_records; ++g)
        for (int32_t r = 0; r < reads_per_record[g]; ++r, ++i) {
            seen.set(bucket_of_host(read_lengths[i], tables_[0].rules));
            weight += (read_lengths[i] > 640 ? 8 : 1) * (int64_t)std::max(haps_per_record[g], 0);
        }
    if (weight > kSmallPairs * (int64_t)seen.count()) return;
    table_ = &tables_[1];
    fp64_ = &fp64_tables_[1];
}

pairhmm_status_t Engine::build_index(const pairhmm_batch_t& b, const std::vector<TileRule>& rules,
                                     const Fp64Table& fp64, BatchIndex& x, std::string& err) {
    // Scalars reset; vectors keep their storage between calls (an engine
    // reuses one index, so a batch of the same size touches no fresh pages).
    x.num_records = x.num_reads = x.num_haps = x.num_pairs = x.cells = 0;
    x.max_read_len = x.max_hap_len = 0;
    x.read_bytes = x.hap_bytes = x.read_min = x.hap_min = 0;
    x.pack_positions = x.code_bytes = 0;
    x.multi_tile_pairs = 0;
    for (int64_t& c : x.class_pairs) c = 0;
    for (int64_t& c : x.list_start) c = 0;
    x.unit_read0.clear();
    x.unit_read1.clear();
    x.unit_bucket.clear();
    x.bucket_pairs.assign(rules.size(), 0);
    x.bucket_items.assign(rules.size(), 0);
    if (b.num_records < 0) { err = "num_records < 0"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
    x.num_records = b.num_records;
    if (b.num_records == 0) return PAIRHMM_OK;
    if (!b.reads_per_record || !b.haps_per_record) { err = "null record arrays"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
    x.rec_haps.resize(b.num_records);
    x.rec_hap_base.resize(b.num_records);
    x.rec_pair_base.resize(b.num_records);
    for (int64_t g = 0; g < b.num_records; ++g) {
        const int32_t R = b.reads_per_record[g], H = b.haps_per_record[g];
        if (R < 0 || H < 0) { err = "negative reads/haplotypes in a record"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
        x.rec_haps[g] = H;
        x.rec_hap_base[g] = x.num_haps;
        x.rec_pair_base[g] = x.num_pairs;
        x.num_reads += R;
        x.num_haps += H;
        x.num_pairs += (int64_t)R * H;
    }
    if (x.num_reads >= (int64_t(1) << 31) || x.num_haps >= (int64_t(1) << 31)) {
        err = "more than 2^31-1 reads or haplotypes in one batch";
        return PAIRHMM_ERR_INVALID_ARGUMENT;
    }
    if ((x.num_reads && (!b.read_lengths)) || (x.num_haps && !b.hap_lengths)) {
        err = "null length arrays";
        return PAIRHMM_ERR_INVALID_ARGUMENT;
    }
    x.read_record.resize(x.num_reads);
    x.read_local.resize(x.num_reads);
    x.read_start.resize(x.num_reads);
    x.hap_start.resize(x.num_haps);
    x.unit_read0.reserve(x.num_reads);
    x.unit_read1.reserve(x.num_reads);
    x.unit_bucket.reserve(x.num_reads);

    // bucket of every read length up to the longest finite rule, by table
    const int nb = (int)rules.size();
    int lut_max = 0;
    for (const TileRule& r : rules)
        if (r.max_len < (1 << 20)) lut_max = std::max(lut_max, r.max_len);
    std::vector<uint8_t> lut((size_t)lut_max + 1);
    for (int L = 0, bk = 0; L <= lut_max; ++L) {
        while (bk < nb - 1 && L > rules[bk].max_len) ++bk;
        lut[L] = (uint8_t)bk;
    }
    std::vector<uint8_t> packed(nb), multi(nb);
    for (int k = 0; k < nb; ++k) {
        packed[k] = rules[k].packed;
        multi[k] = rules[k].multi_tile;
    }

    // haplotypes: extents, packed starts, per-record length sums
    std::vector<int64_t> rec_hap_sum(b.num_records);
    {
        int64_t h = 0;
        for (int64_t g = 0; g < b.num_records; ++g) {
            int64_t sh = 0;
            for (int32_t k = 0; k < x.rec_haps[g]; ++k, ++h) {
                const int32_t H = b.hap_lengths[h];
                if (H < 1) { err = "haplotype length < 1"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
                if (b.hap_offsets) {
                    const int64_t o = b.hap_offsets[h];
                    if (o < 0) { err = "negative haplotype offset"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
                    x.hap_bytes = std::max<int64_t>(x.hap_bytes, o + H);
                    x.hap_min = h == 0 ? o : std::min<int64_t>(x.hap_min, o);
                }
                x.max_hap_len = std::max(x.max_hap_len, H);
                x.hap_start[h] = x.code_bytes;
                x.code_bytes += round_up(H, 16);
                sh += H;
            }
            rec_hap_sum[g] = sh;
        }
    }

    // reads, one record at a time: record/local index, packed start, bucket
    // counts, and units -- reads of a record in the same bucket, paired when
    // the bucket's kernel is packed (order inside a record does not matter:
    // output slots are per read); cells = sum over records of
    // (sum L) * (sum H) (gpuworker.cuh:495-520)
    std::vector<int32_t> pending(nb, -1);
    std::vector<int> touched;
    touched.reserve(nb);
    int64_t i = 0;
    for (int64_t g = 0; g < b.num_records; ++g) {
        const int64_t H = x.rec_haps[g];
        const int32_t R = b.reads_per_record[g];
        int64_t sl = 0;
        touched.clear();
        for (int32_t r = 0; r < R; ++r, ++i) {
            const int32_t L = b.read_lengths[i];
            if (L < 1) { err = "read length < 1"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
            if (b.read_offsets) {
                const int64_t o = b.read_offsets[i];
                if (o < 0) { err = "negative read offset"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
                x.read_bytes = std::max<int64_t>(x.read_bytes, o + L);
                x.read_min = i == 0 ? o : std::min<int64_t>(x.read_min, o);
            }
            x.max_read_len = std::max(x.max_read_len, L);
            x.read_record[i] = (int32_t)g;
            x.read_local[i] = r;
            x.read_start[i] = x.pack_positions;
            x.pack_positions += round_up(L, 4);
            sl += L;
            const int bk = L <= lut_max ? lut[L] : bucket_of_host(L, rules);
            x.bucket_pairs[bk] += H;
            x.class_pairs[fp64.class_of(L)] += H;
            if (multi[bk]) x.multi_tile_pairs += H;
            if (packed[bk]) {
                if (pending[bk] < 0) {
                    pending[bk] = (int32_t)i;
                    touched.push_back(bk);
                    continue;
                }
                x.unit_read0.push_back(pending[bk]);
                x.unit_read1.push_back((int32_t)i);
                pending[bk] = -1;
            } else {
                x.unit_read0.push_back((int32_t)i);
                x.unit_read1.push_back(-1);
            }
            x.unit_bucket.push_back(bk);
            x.bucket_items[bk] += H;
        }
        for (int bk : touched)
            if (pending[bk] >= 0) {
                x.unit_read0.push_back(pending[bk]);
                x.unit_read1.push_back(-1);
                x.unit_bucket.push_back(bk);
                x.bucket_items[bk] += H;
                pending[bk] = -1;
            }
        x.cells += sl * rec_hap_sum[g];
    }
    {
        int64_t off = 0;
        for (size_t c = 0; c < fp64.classes.size(); ++c) {
            if ((int)c == fp64.exts[fp64.classes[c].ext].first) x.list_start[kMaxFp64Classes + fp64.classes[c].ext] = off;
            x.list_start[c] = off;
            off += x.class_pairs[c];
        }
    }
    return PAIRHMM_OK;
}

pairhmm_status_t Engine::scan_inputs(const pairhmm_batch_t& b, InputRanges& r, std::string& err, bool gcp) {
    r = InputRanges{};
    if (b.num_records < 0) { err = "num_records < 0"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
    if (b.num_records == 0) return PAIRHMM_OK;
    if (!b.reads_per_record || !b.haps_per_record) { err = "null record arrays"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
    for (int64_t g = 0; g < b.num_records; ++g) {
        const int32_t R = b.reads_per_record[g], H = b.haps_per_record[g];
        if (R < 0 || H < 0) { err = "negative reads/haplotypes in a record"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
        r.num_reads += R;
        r.num_haps += H;
        r.num_pairs += (int64_t)R * H;
    }
    if (r.num_reads >= (int64_t(1) << 31) || r.num_haps >= (int64_t(1) << 31)) {
        err = "more than 2^31-1 reads or haplotypes in one batch";
        return PAIRHMM_ERR_INVALID_ARGUMENT;
    }
    if (r.num_reads > 0 && (!b.read_lengths || !b.read_offsets || !b.read_bases || !b.base_quals || !b.ins_quals ||
                            !b.del_quals)) {
        err = "null read arrays";
        return PAIRHMM_ERR_INVALID_ARGUMENT;
    }
    if (r.num_haps > 0 && (!b.hap_lengths || !b.hap_offsets || !b.hap_bases)) {
        err = "null haplotype arrays";
        return PAIRHMM_ERR_INVALID_ARGUMENT;
    }
    if (gcp && r.num_reads > 0 && !b.gcp_quals) {
        err = "gcp mode needs the gcp quality array";
        return PAIRHMM_ERR_INVALID_ARGUMENT;
    }
    for (int64_t i = 0; i < r.num_reads; ++i) {
        const int32_t L = b.read_lengths[i];
        const int64_t o = b.read_offsets[i];
        if (L < 1) { err = "read length < 1"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
        if (o < 0) { err = "negative read offset"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
        if (gcp && b.gcp_quals[o] == 0) {
            err = "gcp quality 0 (eps = 1, beta = 0) has no gap-to-match transition to rescale by";
            return PAIRHMM_ERR_INVALID_ARGUMENT;
        }
        r.read_min = i == 0 ? o : std::min(r.read_min, o);
        r.read_end = std::max(r.read_end, o + L);
    }
    for (int64_t h = 0; h < r.num_haps; ++h) {
        const int32_t H = b.hap_lengths[h];
        const int64_t o = b.hap_offsets[h];
        if (H < 1) { err = "haplotype length < 1"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
        if (o < 0) { err = "negative haplotype offset"; return PAIRHMM_ERR_INVALID_ARGUMENT; }
        r.hap_min = h == 0 ? o : std::min(r.hap_min, o);
        r.hap_end = std::max(r.hap_end, o + H);
    }
    return PAIRHMM_OK;
}

pairhmm_status_t Engine::ensure_inputs(const InputRanges& r) {
    const int64_t nr = std::max<int64_t>(r.num_reads, 1), nh = std::max<int64_t>(r.num_haps, 1);
    const int64_t rb = std::max<int64_t>(r.read_end - r.read_min, 1);
    const int64_t hb = std::max<int64_t>(r.hap_end - r.hap_min, 1);
    PHMM_CUDA(in_read_bases_.ensure(rb));
    PHMM_CUDA(in_bq_.ensure(rb));
    PHMM_CUDA(in_iq_.ensure(rb));
    PHMM_CUDA(in_dq_.ensure(rb));
    if (opts_.gcp) PHMM_CUDA(in_gq_.ensure(rb));
    PHMM_CUDA(in_read_off_.ensure(8 * nr));
    PHMM_CUDA(in_read_len_.ensure(4 * nr));
    PHMM_CUDA(in_hap_bases_.ensure(hb));
    PHMM_CUDA(in_hap_off_.ensure(8 * nh));
    PHMM_CUDA(in_hap_len_.ensure(4 * nh));
    PHMM_CUDA(scores_.ensure(4 * std::max<int64_t>(r.num_pairs, 1)));
    return PAIRHMM_OK;
}

pairhmm_status_t Engine::ensure_buffers(const BatchIndex& x) {
    const int64_t nr = std::max<int64_t>(x.num_reads, 1), np = std::max<int64_t>(x.num_pairs, 1);
    if (opts_.gcp) PHMM_CUDA(read_gcp_.ensure(nr));
    PHMM_CUDA(read_pack_.ensure(4 * (x.pack_positions + kReadSlackPos)));
    PHMM_CUDA(read_meta_.ensure(sizeof(ReadMeta) * nr));
    PHMM_CUDA(hap_code_.ensure(x.code_bytes + kHapSlack));
    const int64_t nbins = (int64_t)table_->rules.size() * hbins_of(x);
    PHMM_CUDA(hist_.ensure(4 * nbins));
    PHMM_CUDA(cursor_.ensure(8 * nbins));
    PHMM_CUDA(items_.ensure(sizeof(Item) * np));
    PHMM_CUDA(rescue_.ensure(sizeof(Task) * np));  // class lists laid out back to back
    PHMM_CUDA(rescue_ext_.ensure(sizeof(Task) * np));  // the extended tier's, same offsets
    return PAIRHMM_OK;
}

namespace {
// The index's arrays: where each one's device pointer goes, its host data and bytes.
struct IndexArray {
    const void** ptr;
    const void* src;
    size_t bytes;
};
}  // namespace

#define PHMM_INDEX_ARRAYS(x)                                                                        \
    {                                                                                               \
        {(const void**)&ix_.read_record, x.read_record.data(), 4 * x.read_record.size()},           \
        {(const void**)&ix_.read_local, x.read_local.data(), 4 * x.read_local.size()},              \
        {(const void**)&ix_.rec_haps, x.rec_haps.data(), 4 * x.rec_haps.size()},                    \
        {(const void**)&ix_.rec_hap_base, x.rec_hap_base.data(), 8 * x.rec_hap_base.size()},        \
        {(const void**)&ix_.rec_pair_base, x.rec_pair_base.data(), 8 * x.rec_pair_base.size()},     \
        {(const void**)&ix_.read_start, x.read_start.data(), 8 * x.read_start.size()},              \
        {(const void**)&ix_.hap_start, x.hap_start.data(), 8 * x.hap_start.size()},                 \
        {(const void**)&ix_.unit_read0, x.unit_read0.data(), 4 * x.unit_read0.size()},              \
        {(const void**)&ix_.unit_read1, x.unit_read1.data(), 4 * x.unit_read1.size()},              \
        {(const void**)&ix_.unit_bucket, x.unit_bucket.data(), 4 * x.unit_bucket.size()},           \
        {(const void**)&ix_.list_start, x.list_start, sizeof(x.list_start)},                        \
    }

pairhmm_status_t Engine::upload_index(const BatchIndex& x, cudaStream_t s) {
    if ((size_t)index_bytes(x) + sizeof(x.list_start) <= HostUploader::kGatherBytes / 2)
        return upload_gathered(x, nullptr, nullptr, s);
    DevBuf* const bufs[] = {&read_record_,  &read_local_, &rec_haps_,   &rec_hap_base_, &rec_pair_base_, &read_start_,
                            &hap_start_,    &unit_read0_, &unit_read1_, &unit_bucket_,  &rescue_off_};
    const IndexArray arrays[] = PHMM_INDEX_ARRAYS(x);
    static_assert(sizeof(bufs) / sizeof(bufs[0]) == sizeof(arrays) / sizeof(arrays[0]), "a buffer per array");
    std::vector<HostUploader::Copy> copies;
    for (size_t i = 0; i < sizeof(arrays) / sizeof(arrays[0]); ++i) {
        PHMM_CUDA(bufs[i]->ensure(std::max<size_t>(arrays[i].bytes, 1)));
        *arrays[i].ptr = bufs[i]->ptr;
        copies.push_back({bufs[i]->ptr, arrays[i].src, arrays[i].bytes});
    }
    PHMM_CUDA(uploader_.run(opts_.device, copies, s));
    return PAIRHMM_OK;
}

size_t Engine::input_bytes(const InputRanges& r, bool gcp) {
    return (size_t)((gcp ? 5 : 4) * (r.read_end - r.read_min) + (r.hap_end - r.hap_min) + 12 * r.num_reads +
                    12 * r.num_haps);
}

pairhmm_status_t Engine::upload_gathered(const BatchIndex& x, const InputRanges* r, pairhmm_batch_t* in,
                                         cudaStream_t s) {
    const IndexArray index[] = PHMM_INDEX_ARRAYS(x);
    std::vector<HostUploader::Part> parts;
    parts.reserve(24);
    std::vector<const void**> ptrs;
    ptrs.reserve(24);
    size_t total = 0;
    auto add = [&](const void** ptr, const void* src, size_t bytes) {
        parts.push_back({total, src, bytes});
        ptrs.push_back(ptr);
        total += (bytes + 15) & ~size_t(15);
    };
    if (r) {
        const size_t rn = (size_t)(r->read_end - r->read_min), hn = (size_t)(r->hap_end - r->hap_min);
        add((const void**)&in->read_bases, in->read_bases + r->read_min, rn);
        add((const void**)&in->base_quals, in->base_quals + r->read_min, rn);
        add((const void**)&in->ins_quals, in->ins_quals + r->read_min, rn);
        add((const void**)&in->del_quals, in->del_quals + r->read_min, rn);
        if (opts_.gcp) add((const void**)&in->gcp_quals, in->gcp_quals + r->read_min, rn);
        add((const void**)&in->hap_bases, in->hap_bases + r->hap_min, hn);
        add((const void**)&in->read_offsets, in->read_offsets, 8 * (size_t)r->num_reads);
        add((const void**)&in->read_lengths, in->read_lengths, 4 * (size_t)r->num_reads);
        add((const void**)&in->hap_offsets, in->hap_offsets, 8 * (size_t)r->num_haps);
        add((const void**)&in->hap_lengths, in->hap_lengths, 4 * (size_t)r->num_haps);
    }
    for (const IndexArray& a : index) add(a.ptr, a.src, a.bytes);
    PHMM_CUDA(arena_.ensure(total));
    PHMM_CUDA(uploader_.gather(opts_.device, arena_.ptr, total, parts, s));
    for (size_t i = 0; i < ptrs.size(); ++i) *ptrs[i] = arena_.as<uint8_t>() + parts[i].offset;
    if (r) {
        // the caller's absolute offsets stay valid: byte arrays are shifted to their start
        auto shift = [](const uint8_t*& p, int64_t lo) {
            p = reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(p) - (uintptr_t)lo);
        };
        shift(in->read_bases, r->read_min);
        shift(in->base_quals, r->read_min);
        shift(in->ins_quals, r->read_min);
        shift(in->del_quals, r->read_min);
        if (opts_.gcp) shift(in->gcp_quals, r->read_min);
        shift(in->hap_bases, r->hap_min);
    }
    return PAIRHMM_OK;
}

// haplotype-length classes of a batch's work list (prep_kernels.cuh)
int64_t Engine::hbins_of(const BatchIndex& x) const {
    return opts_.mode == PAIRHMM_MODE_PLAIN ? 4 : round_up((int64_t)std::min(kHBins - 1, x.max_hap_len) + 1, 4);
}

int64_t Engine::index_bytes(const BatchIndex& x) {
    return 4 * (int64_t)(x.read_record.size() + x.read_local.size() + x.rec_haps.size() + x.unit_read0.size() +
                         x.unit_read1.size() + x.unit_bucket.size()) +
           8 * (int64_t)(x.rec_hap_base.size() + x.rec_pair_base.size() + x.read_start.size() + x.hap_start.size());
}

// A kernel's shared memory opt-in and occupancy, which load its code (about 0.4 ms in a
// process that has not used it).
pairhmm_status_t Engine::load_kernel(const void* kernel, int threads, size_t smem) {
    if (blocks_per_sm_.count(kernel)) return PAIRHMM_OK;
    int per_sm = 0;
    PHMM_CUDA(cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    PHMM_CUDA(cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem));
    blocks_per_sm_.emplace(kernel, std::max(per_sm, 1));
    return PAIRHMM_OK;
}

// The kernels a batch on these tables launches, or (x null) could launch.  A batch's own
// are loaded ahead of its plan: creating an engine with all 200 of both tables takes 90 ms
// in a fresh process, 14 ms without.
pairhmm_status_t Engine::load_kernels(const TileTable& table, const Fp64Table& fp64, const BatchIndex* x) {
    pairhmm_status_t st = PAIRHMM_OK;
    auto load = [&](const auto* c) {
        if (st == PAIRHMM_OK) st = load_kernel(c->kernel, c->block_threads, c->smem_bytes);
    };
    for (size_t b = 0; b < table.cfg.size(); ++b)
        if (!x || x->bucket_items[b] != 0) load(table.cfg[b]);
    for (size_t c = 0; c < fp64.classes.size(); ++c) {
        if (x && x->class_pairs[c] == 0) continue;
        load(fp64.classes[c].scaled);
        load(fp64.exts[fp64.classes[c].ext].cfg);
        if (c + 1 == fp64.classes.size()) load(fp64.fused);
    }
    return st;
}

pairhmm_status_t Engine::load_all() {
    PHMM_CUDA(cudaSetDevice(opts_.device));
    for (int i = 0; i < 2; ++i) {
        const pairhmm_status_t st = load_kernels(tables_[i], fp64_tables_[i], nullptr);
        if (st != PAIRHMM_OK) return st;
    }
    return ensure_side_streams(kSideStreams);
}

// The grid of a persistent launch: every block that fits at once.
int Engine::persistent_grid(const void* kernel) const { return blocks_per_sm_.at(kernel) * num_sms_; }

pairhmm_status_t Engine::enqueue_pipeline(const pairhmm_batch_t& in, const BatchIndex& x, const Plan& plan,
                                          float* d_scores, cudaStream_t s, int stage) {
    const int nb = (int)table_->rules.size();
    const bool plain = opts_.mode == PAIRHMM_MODE_PLAIN;
    const int prep_grid = 4 * num_sms_;

    PrepArgs pa{};
    pa.read_bases = in.read_bases;
    pa.base_quals = in.base_quals;
    pa.ins_quals = in.ins_quals;
    pa.del_quals = in.del_quals;
    pa.read_offsets = in.read_offsets;
    pa.read_lengths = in.read_lengths;
    pa.hap_bases = in.hap_bases;
    pa.hap_offsets = in.hap_offsets;
    pa.hap_lengths = in.hap_lengths;
    pa.gcp_quals = opts_.gcp ? in.gcp_quals : nullptr;
    pa.read_gcp = opts_.gcp ? read_gcp_.as<uint8_t>() : nullptr;
    pa.read_record = ix_.read_record;
    pa.read_local = ix_.read_local;
    pa.rec_haps = ix_.rec_haps;
    pa.rec_hap_base = ix_.rec_hap_base;
    pa.rec_pair_base = ix_.rec_pair_base;
    pa.read_start = ix_.read_start;
    pa.hap_start = ix_.hap_start;
    pa.num_reads = x.num_reads;
    pa.num_haps = x.num_haps;
    pa.read_pack = read_pack_.as<uint32_t>();
    pa.hap_code = hap_code_.as<uint8_t>();
    pa.read_meta = read_meta_.as<ReadMeta>();
    pa.ph2pr = ph2pr_.as<float>();
    if (stage == 0) {
    launches_ = 0;
    fp32_launches_ = 0;
    // zero the histogram and the work/rescue counters, pad the haplotype codes, and
    // pack the inputs, in one launch
    FillArgs fa{};
    fa.ptr[0] = reinterpret_cast<uint32_t*>(hap_code_.as<uint8_t>() + x.code_bytes);  // 16-byte aligned
    fa.words[0] = kHapSlack / 4;
    fa.value[0] = 0x04040404u;
    fa.ptr[1] = hist_.as<uint32_t>();
    fa.words[1] = (long long)nb * hbins_of(x);
    fa.ptr[2] = counters_.as<uint32_t>();
    fa.words[2] = 2 * kCtrTotal;
    fa.ptr[3] = rsort_.as<uint32_t>();
    fa.words[3] = (long long)fp64_->classes.size() * kRescueHBins;
    PHMM_CUDA(launch_pack(pa, fa, prep_grid, s));
    launches_ += 1;
    }

    BinArgs ba{};
    ba.hap_lengths = in.hap_lengths;
    ba.read_record = pa.read_record;
    ba.read_local = pa.read_local;
    ba.rec_haps = pa.rec_haps;
    ba.rec_hap_base = pa.rec_hap_base;
    ba.rec_pair_base = pa.rec_pair_base;
    ba.unit_read0 = ix_.unit_read0;
    ba.unit_read1 = ix_.unit_read1;
    ba.unit_bucket = ix_.unit_bucket;
    ba.num_units = (int64_t)x.unit_read0.size();
    ba.nbuckets = nb;
    ba.hcap = plain ? 0 : std::min(kHBins - 1, x.max_hap_len);
    ba.hbins = (int)hbins_of(x);
    for (int rank = 0; rank < nb; ++rank)
        ba.ranks.begin[rank + 1] = ba.ranks.begin[rank] + x.bucket_items[plain ? rank : nb - 1 - rank];
    ba.reversed = !plain;
    ba.hist = hist_.as<unsigned int>();
    ba.cursor = cursor_.as<unsigned long long>();
    ba.items = items_.as<Item>();
    if (stage == 0) {
    PHMM_CUDA(launch_binning(ba, prep_grid, s));
    launches_ += 3;
    return PAIRHMM_OK;
    }

    unsigned long long* counters = counters_.as<unsigned long long>();
    DevView v{};
    v.read_pack = pa.read_pack;
    v.read_meta = pa.read_meta;
    v.read_start = pa.read_start;
    v.read_len = in.read_lengths;
    v.hap_code = pa.hap_code;
    v.hap_start = pa.hap_start;
    v.hap_len = in.hap_lengths;
    v.scores = d_scores;
    v.rescue_base = rescue_.as<Task>();
    v.rescue_class = fp64_lut_[fp64_ == &fp64_tables_[1]].as<uint8_t>();
    v.rescue_off = ix_.list_start;
    v.rescue_count = counters + kCtrScaled;
    v.rescue_enabled = (!plain && opts_.fp64_rescue) ? 1 : 0;
    v.ph2pr = ph2pr_.as<float>();
    v.read_gcp = pa.read_gcp;

    // FP64 pass: first sort each class's list by haplotype length into the
    // work-item buffer (free once the FP32 stage is done), same class offsets
    const int64_t upper = x.num_pairs;  // pairs the FP64 lists could hold
    const bool sorted = fp64_warps(x) > kNoSortWarps;
    Task* const fp64_lists = sorted ? items_.as<Task>() : rescue_.as<Task>();
    if (stage == 2 && sorted) {
        RescueSortArgs ra{};
        ra.in = rescue_.as<Task>();
        ra.out = fp64_lists;
        ra.classes = (int)fp64_->classes.size();
        ra.off = ix_.list_start;
        ra.count = counters + kCtrScaled;
        ra.hap_len = in.hap_lengths;
        ra.hist = rsort_.as<unsigned int>();
        ra.cursor = reinterpret_cast<unsigned long long*>(rsort_.as<unsigned int>() + kMaxFp64Classes * kRescueHBins);
        const int sort_grid = (int)std::max<int64_t>(1, std::min<int64_t>((upper + 255) / 256, 8 * (int64_t)num_sms_));
        PHMM_CUDA(launch_rescue_sort(ra, sort_grid, s));
        launches_ += 3;
    }

    // engine form: the stage's launches go round-robin onto the side streams
    // (forked from s, joined back below); the plain form, and a single launch, keep s
    const int nside = plan.side[stage];
    int nlaunch = 0;
    auto next_stream = [&]() { return nside ? side_[nlaunch++ % nside] : s; };
    // staged_: the host waits in the streams' place
    auto fork = [&]() {
        if (nside && staged_) PHMM_CUDA(cudaStreamSynchronize(s));
        if (!nside || staged_) return PAIRHMM_OK;
        PHMM_CUDA(cudaEventRecord(fork_, s));
        for (int i = 0; i < nside; ++i) PHMM_CUDA(cudaStreamWaitEvent(side_[i], fork_, 0));
        return PAIRHMM_OK;
    };
    auto join = [&]() {
        for (int i = 0; i < nside; ++i) {
            if (staged_) {
                PHMM_CUDA(cudaStreamSynchronize(side_[i]));
                continue;
            }
            PHMM_CUDA(cudaEventRecord(join_[i], side_[i]));
            PHMM_CUDA(cudaStreamWaitEvent(s, join_[i], 0));
        }
        return PAIRHMM_OK;
    };
    pairhmm_status_t fs = fork();
    if (fs != PAIRHMM_OK) return fs;
    if (stage == 1) {
        for (int rank = 0; rank < nb; ++rank) {
            const int b = plain ? rank : nb - 1 - rank;
            if (x.bucket_items[b] == 0) continue;
            const ConfigInfo* c = table_->cfg[b];
            Fp32LaunchArgs la{};
            la.view = v;
            la.items = items_.as<Item>() + ba.ranks.begin[rank];
            la.num_items = x.bucket_items[b];
            la.persistent = plan.persistent[b];
            la.counter = counters + rank;
            la.scratch = static_cast<char*>(scratch_.ptr) + plan.scratch_off[b];
            la.rows = plan.rows;
            la.grid = plan.grid[b];
            la.stream = next_stream();
            PHMM_CUDA(c->launch(la));
            ++launches_;
            ++fp32_launches_;
        }
    } else {
        // stage 2: FP64 pass over flagged pairs (FP32 underflow, or degenerate alpha):
        // per length class the scaled tier, then the extended tier over the pairs the
        // scaled tier handed on.  An extended class that serves one scaled class runs
        // right behind it on the same stream (for the padded multi-tile class of a small
        // batch, inside the scaled tier's launch); the others once all scaled launches
        // are done.
        auto launch = [&](const Fp64Config* cfg, bool tier_ext, int list, int grid, int64_t scratch, int ext_cls,
                          cudaStream_t on) {
            Fp64LaunchArgs fa{};
            fa.view = v;
            fa.ext_list = {rescue_ext_.as<Task>(), ix_.list_start + kMaxFp64Classes, counters + kCtrExt,
                           ext_cls};
            fa.items = (tier_ext ? rescue_ext_.as<Task>() : fp64_lists) +
                       x.list_start[tier_ext ? kMaxFp64Classes + list : list];
            fa.count = counters + (tier_ext ? kCtrExt : kCtrScaled) + list;
            fa.counter = counters + (tier_ext ? kCtrTaskExt : kCtrTaskScaled) + list;
            fa.scratch = static_cast<char*>(scratch_.ptr) + scratch;
            fa.rows = plan.rows;
            fa.grid = grid;
            fa.stream = on;
            ++launches_;
            return cfg->launch(fa);
        };
        const int last = (int)fp64_->classes.size() - 1;
        bool shared_ext[kMaxFp64Classes] = {};
        std::vector<std::pair<cudaStream_t, int>> behind;
        for (int c = last; c >= 0; --c) {
            if (x.class_pairs[c] == 0) continue;
            const Fp64Table::Class& k = fp64_->classes[c];
            const Fp64Table::Ext& e = fp64_->exts[k.ext];
            const cudaStream_t on = next_stream();
            // a few long pairs (at most a round of resident warps): one pass instead of two
            const bool fuse = c == last && x.class_pairs[c] <= kFuseMaxPairs;
            PHMM_CUDA(launch(fuse ? fp64_->fused : k.scaled, false, c, plan.fp64_grid[c], plan.fp64_scratch[c], k.ext,
                             on));
            if (!e.own_stream) shared_ext[k.ext] = true;
            else if (!fuse && staged_ && nside) behind.push_back({on, k.ext});
            else if (!fuse)
                PHMM_CUDA(launch(e.cfg, true, k.ext, plan.fp64_ext_grid[k.ext], plan.fp64_ext_scratch[k.ext], 0, on));
        }
        while (!behind.empty()) {   // staged_: an extended class once its stream's scaled class is done
            const size_t waiting = behind.size();
            for (size_t i = 0; i < behind.size();) {
                const cudaError_t q = cudaStreamQuery(behind[i].first);
                if (q == cudaErrorNotReady) {
                    cudaGetLastError();
                    ++i;
                    continue;
                }
                PHMM_CUDA(q);
                const int e = behind[i].second;
                PHMM_CUDA(launch(fp64_->exts[e].cfg, true, e, plan.fp64_ext_grid[e], plan.fp64_ext_scratch[e], 0,
                                 behind[i].first));
                behind.erase(behind.begin() + i);
            }
            if (behind.size() == waiting) std::this_thread::yield();
        }
        bool any = false;
        for (bool b : shared_ext) any = any || b;
        if (any) {
            if ((fs = join()) != PAIRHMM_OK || (fs = fork()) != PAIRHMM_OK) return fs;
            for (int e = 0; e < (int)fp64_->exts.size(); ++e)
                if (shared_ext[e])
                    PHMM_CUDA(launch(fp64_->exts[e].cfg, true, e, plan.fp64_ext_grid[e], plan.fp64_ext_scratch[e], 0,
                                     next_stream()));
        }
    }
    return join();
}

Engine::Plan Engine::make_plan(const BatchIndex& x) const {
    const int nb = (int)table_->rules.size();
    const bool plain = opts_.mode == PAIRHMM_MODE_PLAIN;
    Plan p;
    p.rows = round_up((int64_t)x.max_hap_len + 2 * 32 + 8, 64);
    p.grid.assign(nb, 0);
    p.persistent.assign(nb, 1);
    p.scratch_off.assign(nb, 0);
    // multi-tile buckets may run at the same time: each gets its own slice of
    // the border scratch, out of an equal share of the budget
    int n_mt = 0;
    for (int b = 0; b < nb; ++b)
        if (x.bucket_items[b] != 0 && table_->cfg[b]->scratch_bytes_per_row) ++n_mt;
    const int64_t mt_budget = kScratchBudget / std::max(1, n_mt);
    int64_t scratch = 0, fp32_scratch = 0;
    for (int b = 0; b < nb; ++b) {
        if (x.bucket_items[b] == 0) continue;
        const ConfigInfo* c = table_->cfg[b];
        const int64_t tasks = (x.bucket_items[b] + c->per_task - 1) / c->per_task;
        const int64_t need_blocks = (tasks + c->tasks_per_block - 1) / c->tasks_per_block;
        const int64_t resident = persistent_grid(c->kernel);
        int64_t grid = plain ? need_blocks : std::min(resident, need_blocks);
        if (c->scratch_bytes_per_row) {
            const int64_t per_warp = (int64_t)c->scratch_bytes_per_row * p.rows;
            const int64_t cap_blocks = std::max<int64_t>(1, mt_budget / (per_warp * kWarpsPerBlock));
            grid = std::min(grid, cap_blocks);
            p.scratch_off[b] = fp32_scratch;
            fp32_scratch += round_up(grid * kWarpsPerBlock * per_warp, 256);
        }
        grid = std::max<int64_t>(1, std::min<int64_t>(grid, INT32_MAX));
        p.grid[b] = (int)grid;
        // the plain form runs one task per warp; a grid capped by scratch loops on the counter
        p.persistent[b] = (!plain || grid < need_blocks) ? 1 : 0;
    }
    // FP64 launches: no more blocks than the class's pairs could need.  Kernels with
    // border scratch may run at the same time, so each has its own slice, out of an
    // equal share of the budget; an extended class of one scaled class runs behind it
    // and shares its slice.
    int n_scratch = 0;
    for (size_t c = 0; c < fp64_->classes.size(); ++c)
        if (x.class_pairs[c] > 0) n_scratch += fp64_->classes[c].scaled->scratch_bytes_per_row > 0;
    for (const Fp64Table::Ext& e : fp64_->exts) n_scratch += e.cfg->scratch_bytes_per_row > 0 && !e.own_stream;
    auto fp64_grid = [&](const Fp64Config* c, int64_t pairs, int64_t& bytes) {
        const int64_t tasks = (pairs + c->per_task - 1) / c->per_task;
        int64_t grid = std::min<int64_t>(persistent_grid(c->kernel),
                                         (tasks + c->tasks_per_block - 1) / c->tasks_per_block);
        grid = std::max<int64_t>(grid, 1);
        bytes = 0;
        if (c->scratch_bytes_per_row) {
            const int64_t per_block = (int64_t)c->scratch_bytes_per_row * p.rows * c->tasks_per_block;
            grid = std::min(grid, std::max<int64_t>(1, kScratchBudget / std::max(1, n_scratch) / per_block));
            bytes = round_up(grid * per_block, 256);
        }
        return (int)grid;
    };
    for (size_t i = 0; i < fp64_->exts.size(); ++i) {
        const Fp64Table::Ext& e = fp64_->exts[i];
        int64_t pairs = 0, slice = 0, bytes = 0;
        for (int c = e.first; c <= e.last; ++c) {
            if (x.class_pairs[c] == 0) continue;
            pairs += x.class_pairs[c];
            const Fp64Config* scaled = fp64_->classes[c].scaled;
            p.fp64_scratch[c] = scratch;
            p.fp64_grid[c] = fp64_grid(scaled, x.class_pairs[c], bytes);
            if (e.own_stream) slice = bytes;
            else scratch += bytes;
        }
        if (pairs == 0) continue;
        p.fp64_ext_scratch[i] = scratch;
        p.fp64_ext_grid[i] = fp64_grid(e.cfg, pairs, bytes);
        scratch += std::max(slice, bytes);
    }
    p.scratch_bytes = (size_t)std::max<int64_t>(std::max(scratch, fp32_scratch), 256);
    int launches[3] = {};
    for (int b = 0; b < nb; ++b) launches[1] += x.bucket_items[b] != 0;
    for (int64_t n : x.class_pairs) launches[2] += n != 0;
    for (int st = 1; st < 3; ++st) p.side[st] = plain || launches[st] < 2 ? 0 : std::min(launches[st], kSideStreams);
    return p;
}

// Warps of the FP64 groups that the batch's pairs could take, a narrower group counting as one.
int64_t Engine::fp64_warps(const BatchIndex& x) const {
    int64_t warps = 0;
    for (size_t c = 0; c < fp64_->classes.size(); ++c)
        warps += x.class_pairs[c] * std::max(fp64_->classes[c].scaled->G / 32, 1);
    return warps;
}

// What decides a batch's launches and their dependencies (not their arguments).
std::vector<uint8_t> Engine::launch_shape(const BatchIndex& x, const Plan& plan) const {
    std::vector<uint8_t> shape = {(uint8_t)(table_ == &tables_[1]), (uint8_t)(fp64_warps(x) > kNoSortWarps),
                                  (uint8_t)plan.side[1], (uint8_t)plan.side[2]};
    for (const int64_t n : x.bucket_items) shape.push_back(n != 0);
    for (const int64_t n : x.class_pairs) shape.push_back(n != 0);
    shape.push_back(x.class_pairs[fp64_->classes.size() - 1] <= kFuseMaxPairs);
    return shape;
}

pairhmm_status_t Engine::run_pipeline(const pairhmm_batch_t& in, const BatchIndex& x, float* d_scores,
                                      cudaStream_t s) {
    if (x.num_pairs == 0) return PAIRHMM_OK;
    // every buffer the launches reference exists before capture starts
    const pairhmm_status_t loaded = load_kernels(*table_, *fp64_, &x);
    if (loaded != PAIRHMM_OK) return loaded;
    const Plan plan = make_plan(x);
    const pairhmm_status_t side = ensure_side_streams(std::max(plan.side[1], plan.side[2]));
    if (side != PAIRHMM_OK) return side;
    PHMM_CUDA(scratch_.ensure(plan.scratch_bytes));
    const cudaEvent_t marks[3] = {ev_prep_, ev_fp32_, ev1_};
    // A graph only for small batches that launch the same kernels as the kept graph, or as
    // the eight batches before: instantiating one costs more than its 7-37 launches, and
    // mixed small batches rarely have the same length classes (changing batches of uneven
    // regions, graph / launches a call: 4 regions 0.65 / 0.30 ms, 24 regions 1.57 / 0.67).
    // And only for few classes: the same batch again, classes of 96-4,000 pairs in all,
    // graph over launches: 1-3 classes 0.91-1.0, 4-6 0.92-1.03, 8 0.96-1.2, 10 1.05-1.18,
    // 12 1.0-1.13.
    bool use_graph = false;
    if (opts_.use_graphs && !staged_ && x.num_pairs <= kGraphMaxPairs && plan.side[1] <= kGraphMaxClasses) {
        std::vector<uint8_t> shape = launch_shape(x, plan);
        shape_repeats_ = shape == last_shape_ ? shape_repeats_ + 1 : 0;
        use_graph = shape_repeats_ >= kGraphAfter || (graph_exec_ && shape == graph_shape_);
        last_shape_ = std::move(shape);
    }
    if (!use_graph) {
        for (int stage = 0; stage < 3; ++stage) {
            const pairhmm_status_t st = enqueue_pipeline(in, x, plan, d_scores, s, stage);
            if (st != PAIRHMM_OK) return st;
            PHMM_CUDA(cudaEventRecord(marks[stage], s));
        }
        return PAIRHMM_OK;
    }
    // one graph for the three stages, the marks between them recorded by its nodes
    cudaGraph_t graph = nullptr;
    PHMM_CUDA(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    pairhmm_status_t st = PAIRHMM_OK;
    for (int stage = 0; stage < 3 && st == PAIRHMM_OK; ++stage) {
        st = enqueue_pipeline(in, x, plan, d_scores, s, stage);
        if (st != PAIRHMM_OK) break;
        const cudaError_t me = cudaEventRecordWithFlags(marks[stage], s, cudaEventRecordExternal);
        if (me != cudaSuccess) st = cuda_fail(me, "cudaEventRecordWithFlags");
    }
    cudaError_t ce = cudaStreamEndCapture(s, &graph);
    if (st != PAIRHMM_OK) {
        if (graph) cudaGraphDestroy(graph);
        return st;
    }
    if (ce != cudaSuccess) return cuda_fail(ce, "cudaStreamEndCapture");
    if (graph_exec_) {
        cudaGraphExecUpdateResultInfo info{};
        if (cudaGraphExecUpdate(graph_exec_, graph, &info) != cudaSuccess) {
            cudaGetLastError();
            cudaGraphExecDestroy(graph_exec_);
            graph_exec_ = nullptr;
        }
    }
    if (!graph_exec_) {
        ce = cudaGraphInstantiate(&graph_exec_, graph, 0);
        if (ce != cudaSuccess) graph_exec_ = nullptr;
    }
    cudaGraphDestroy(graph);
    if (ce != cudaSuccess) return cuda_fail(ce, "cudaGraphInstantiate");
    graph_shape_ = last_shape_;
    PHMM_CUDA(cudaGraphLaunch(graph_exec_, s));
    return PAIRHMM_OK;
}

pairhmm_status_t Engine::host_begin(const pairhmm_batch_t& b, float* scores, cudaEvent_t mark_start,
                                    cudaEvent_t mark_end) {
    PHMM_CUDA(cudaSetDevice(opts_.device));
    // first a cheap validating pass for sizes and byte ranges, so the input
    // upload runs on helper threads while this thread builds the index
    InputRanges rg;
    std::string err;
    pairhmm_status_t st = scan_inputs(b, rg, err, opts_.gcp != 0);
    if (st != PAIRHMM_OK) return fail(st, err);
    if (rg.num_pairs > 0 && !scores) return fail(PAIRHMM_ERR_INVALID_ARGUMENT, "null scores");
    stats_ = pairhmm_stats_t{};
    pending_ = false;
    if (rg.num_pairs == 0) return PAIRHMM_OK;
    cudaStream_t s = stream_;
    choose_table(b.num_records, b.reads_per_record, b.haps_per_record, b.read_lengths, rg.num_pairs);
    const BatchIndex& x = idx_;
    pairhmm_batch_t dev = b;
    // upper bound of what a gathered upload takes, alignment included
    const size_t gathered = input_bytes(rg, opts_.gcp != 0) + 28 * (size_t)rg.num_reads + 8 * (size_t)rg.num_haps +
                            20 * (size_t)b.num_records + sizeof(x.list_start) + 512;
    if (gathered <= HostUploader::kGatherBytes) {
        PHMM_CUDA(scores_.ensure(4 * rg.num_pairs));
        if ((st = build_index(b, table_->rules, *fp64_, idx_, err)) != PAIRHMM_OK) return fail(st, err);
        if ((st = ensure_buffers(x)) != PAIRHMM_OK) return st;
        if ((st = upload_gathered(x, &rg, &dev, s)) != PAIRHMM_OK) return st;
    } else {
        if ((st = ensure_inputs(rg)) != PAIRHMM_OK) return st;
        // only the byte range the batch references is copied; device base pointers
        // are shifted so the caller's absolute offsets stay valid
        const int64_t rlo = rg.read_min, rn = rg.read_end - rg.read_min;
        const int64_t hlo = rg.hap_min, hn = rg.hap_end - rg.hap_min;
        std::vector<HostUploader::Copy> inputs = {
            {in_read_bases_.ptr, b.read_bases + rlo, (size_t)rn},
            {in_bq_.ptr, b.base_quals + rlo, (size_t)rn},
            {in_iq_.ptr, b.ins_quals + rlo, (size_t)rn},
            {in_dq_.ptr, b.del_quals + rlo, (size_t)rn},
            {in_read_off_.ptr, b.read_offsets, (size_t)(8 * rg.num_reads)},
            {in_read_len_.ptr, b.read_lengths, (size_t)(4 * rg.num_reads)},
            {in_hap_bases_.ptr, b.hap_bases + hlo, (size_t)hn},
            {in_hap_off_.ptr, b.hap_offsets, (size_t)(8 * rg.num_haps)},
            {in_hap_len_.ptr, b.hap_lengths, (size_t)(4 * rg.num_haps)},
        };
        if (opts_.gcp) inputs.push_back({in_gq_.ptr, b.gcp_quals + rlo, (size_t)rn});
        cudaError_t up = uploader_.start(opts_.device, inputs, s);
        st = build_index(b, table_->rules, *fp64_, idx_, err);
        const cudaError_t upf = uploader_.finish();
        if (up == cudaSuccess) up = upf;
        if (up != cudaSuccess) return cuda_fail(up, "input upload");
        if (st != PAIRHMM_OK) return fail(st, err);
        if ((st = ensure_buffers(x)) != PAIRHMM_OK) return st;
        if ((st = upload_index(x, s)) != PAIRHMM_OK) return st;

        auto shifted = [](const DevBuf& d, int64_t lo) {
            return reinterpret_cast<const uint8_t*>(reinterpret_cast<uintptr_t>(d.ptr) - (uintptr_t)lo);
        };
        dev.read_bases = shifted(in_read_bases_, rlo);
        dev.base_quals = shifted(in_bq_, rlo);
        dev.ins_quals = shifted(in_iq_, rlo);
        dev.del_quals = shifted(in_dq_, rlo);
        dev.gcp_quals = opts_.gcp ? shifted(in_gq_, rlo) : nullptr;
        dev.read_offsets = in_read_off_.as<int64_t>();
        dev.read_lengths = in_read_len_.as<int32_t>();
        dev.hap_bases = shifted(in_hap_bases_, hlo);
        dev.hap_offsets = in_hap_off_.as<int64_t>();
        dev.hap_lengths = in_hap_len_.as<int32_t>();
    }
    stats_.pairs = x.num_pairs;
    stats_.cells = x.cells;
    stats_.multi_tile_pairs = x.multi_tile_pairs;

    PHMM_CUDA(cudaEventRecord(ev0_, s));
    if (mark_start) PHMM_CUDA(cudaEventRecord(mark_start, s));
    if ((st = run_pipeline(dev, x, scores_.as<float>(), s)) != PAIRHMM_OK) return st;
    if (mark_end) PHMM_CUDA(cudaEventRecord(mark_end, s));
    // rescue counts and (into page-locked memory) scores come down now; scores
    // for pageable memory go through the uploader's slots in host_end
    PHMM_CUDA(cudaMemcpyAsync(host_hdr_, counters_.as<unsigned long long>() + kCtrScaled,
                              sizeof(unsigned long long) * 2 * kMaxFp64Classes, cudaMemcpyDeviceToHost, s));
    pend_direct_ = HostUploader::is_page_locked(scores);
    if (pend_direct_)
        PHMM_CUDA(cudaMemcpyAsync(scores, scores_.ptr, 4 * (size_t)x.num_pairs, cudaMemcpyDeviceToHost, s));
    pend_scores_ = scores;
    pend_pairs_ = x.num_pairs;
    stats_.h2d_bytes = (int64_t)input_bytes(rg, opts_.gcp != 0) + index_bytes(x);
    stats_.d2h_bytes = 4 * x.num_pairs + (int64_t)sizeof(unsigned long long) * 2 * kMaxFp64Classes;
    stats_.launches = launches_;
    stats_.fp32_launches = fp32_launches_;
    pending_ = true;
    return PAIRHMM_OK;
}

pairhmm_status_t Engine::host_end() {
    if (!pending_) return PAIRHMM_OK;
    pending_ = false;
    PHMM_CUDA(cudaSetDevice(opts_.device));
    cudaStream_t s = stream_;
    if (!pend_direct_)
        PHMM_CUDA(uploader_.download(opts_.device, pend_scores_, scores_.ptr, 4 * (size_t)pend_pairs_, s));
    PHMM_CUDA(cudaStreamSynchronize(s));
    // per class: the scaled tier's counts, then the extended tier's
    unsigned long long rescued_by_class[2 * kMaxFp64Classes] = {};
    std::memcpy(rescued_by_class, host_hdr_, sizeof(rescued_by_class));
    float ms = 0.f, a = 0.f, b2 = 0.f, c = 0.f;
    PHMM_CUDA(cudaEventElapsedTime(&ms, ev0_, ev1_));
    PHMM_CUDA(cudaEventElapsedTime(&a, ev0_, ev_prep_));
    PHMM_CUDA(cudaEventElapsedTime(&b2, ev_prep_, ev_fp32_));
    PHMM_CUDA(cudaEventElapsedTime(&c, ev_fp32_, ev1_));
    stats_.device_ms = ms;
    stats_.prep_ms = a;
    stats_.fp32_ms = b2;
    stats_.fp64_ms = c;
    stats_.rescued = 0;
    stats_.rescued_ext = 0;
    for (int c = 0; c < kMaxFp64Classes; ++c) {
        stats_.rescued += (int64_t)rescued_by_class[c];
        stats_.rescued_ext += (int64_t)rescued_by_class[kMaxFp64Classes + c];
    }
    return PAIRHMM_OK;
}

pairhmm_status_t Engine::compute_host(const pairhmm_batch_t& b, float* scores) {
    const auto t0 = std::chrono::steady_clock::now();
    // large batches run as chunks of whole records on this engine and a twin
    // engine in turn, so a chunk's index build and upload overlap the previous
    // chunk's kernels
    int64_t pairs = 0;
    if (b.num_records > 0 && b.reads_per_record && b.haps_per_record)
        for (int64_t g = 0; g < b.num_records; ++g)
            pairs += (int64_t)std::max(b.reads_per_record[g], 0) * std::max(b.haps_per_record[g], 0);
    int nchunks = opts_.pipeline_chunks > 0 ? opts_.pipeline_chunks
                                             : (int)std::min<int64_t>(kMaxChunks, pairs / kChunkPairs);
    if (nchunks > b.num_records) nchunks = (int)b.num_records;
    if (nchunks < 2 || !b.read_lengths || !b.hap_lengths || !b.read_offsets || !b.hap_offsets) {
        pairhmm_status_t st = host_begin(b, scores, nullptr, nullptr);
        if (st == PAIRHMM_OK) st = host_end();
        stats_.total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
        return st;
    }
    if (!twin_) {
        pairhmm_options_t o = opts_;
        o.pipeline_chunks = 1;
        twin_ = std::make_unique<Engine>(o);
        pairhmm_status_t st = twin_->init();
        if (st == PAIRHMM_OK) st = twin_->set_tile_table(tables_[0].rules);
        if (st != PAIRHMM_OK) {
            last_error_ = "twin engine: " + twin_->last_error();
            twin_.reset();
            return st;
        }
    }
    PHMM_CUDA(cudaSetDevice(opts_.device));
    if (!span0_) {
        PHMM_CUDA(cudaEventCreate(&span0_));
        PHMM_CUDA(cudaEventCreate(&span1_));
    }
    // chunk boundaries: records in order, about equal pairs per chunk except the
    // first, which is half a chunk (its index build and upload are not overlapped)
    std::vector<int64_t> bound{0};
    {
        int64_t acc = 0, next = 1;
        for (int64_t g = 0; g < b.num_records && (int)bound.size() < nchunks; ++g) {
            acc += (int64_t)std::max(b.reads_per_record[g], 0) * std::max(b.haps_per_record[g], 0);
            if (acc * (2 * nchunks - 1) >= pairs * (2 * next - 1) && g + 1 < b.num_records) {
                bound.push_back(g + 1);
                ++next;
            }
        }
        bound.push_back(b.num_records);
    }
    pairhmm_stats_t sum{};
    Engine* eng[2] = {this, twin_.get()};
    pairhmm_status_t st = PAIRHMM_OK;
    int64_t read0 = 0, hap0 = 0, pair0 = 0;
    const int n = (int)bound.size() - 1;
    auto collect = [&](Engine* e) {
        const pairhmm_status_t r = e->host_end();
        if (r != PAIRHMM_OK) {
            if (e != this) last_error_ = e->last_error();
            return r;
        }
        const pairhmm_stats_t& x = e->stats_;
        sum.pairs += x.pairs;
        sum.cells += x.cells;
        sum.rescued += x.rescued;
        sum.rescued_ext += x.rescued_ext;
        sum.multi_tile_pairs += x.multi_tile_pairs;
        sum.prep_ms += x.prep_ms;
        sum.fp32_ms += x.fp32_ms;
        sum.fp64_ms += x.fp64_ms;
        sum.launches += x.launches;
        sum.fp32_launches += x.fp32_launches;
        sum.h2d_bytes += x.h2d_bytes;
        sum.d2h_bytes += x.d2h_bytes;
        return PAIRHMM_OK;
    };
    for (int i = 0; i < n && st == PAIRHMM_OK; ++i) {
        Engine* e = eng[i & 1];
        if (i >= 2) st = collect(e);  // this engine's previous chunk
        if (st != PAIRHMM_OK) break;
        const int64_t g0 = bound[i], g1 = bound[i + 1];
        int64_t reads = 0, haps = 0, cp = 0;
        for (int64_t g = g0; g < g1; ++g) {
            reads += std::max(b.reads_per_record[g], 0);
            haps += std::max(b.haps_per_record[g], 0);
            cp += (int64_t)std::max(b.reads_per_record[g], 0) * std::max(b.haps_per_record[g], 0);
        }
        pairhmm_batch_t v = b;
        v.num_records = g1 - g0;
        v.reads_per_record += g0;
        v.haps_per_record += g0;
        v.read_offsets += read0;
        v.read_lengths += read0;
        v.hap_offsets += hap0;
        v.hap_lengths += hap0;
        st = e->host_begin(v, scores + pair0, i == 0 ? span0_ : nullptr, i == n - 1 ? span1_ : nullptr);
        if (st != PAIRHMM_OK && e != this) last_error_ = e->last_error();
        read0 += reads;
        hap0 += haps;
        pair0 += cp;
    }
    // the last chunks in flight (also after an error: nothing may stay queued)
    for (int i = std::max(0, n - 2); i < n; ++i) {
        const pairhmm_status_t r = collect(eng[i & 1]);
        if (st == PAIRHMM_OK) st = r;
    }
    if (st != PAIRHMM_OK) return st;
    float span = 0.f;
    PHMM_CUDA(cudaEventElapsedTime(&span, span0_, span1_));
    sum.device_ms = span;
    sum.total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    stats_ = sum;
    return PAIRHMM_OK;
}

pairhmm_status_t Engine::compute_device(const pairhmm_batch_t& b, int32_t, int32_t, float* scores,
                                        cudaStream_t stream) {
    const auto t0 = std::chrono::steady_clock::now();
    PHMM_CUDA(cudaSetDevice(opts_.device));
    if (b.num_records < 0) return fail(PAIRHMM_ERR_INVALID_ARGUMENT, "num_records < 0");
    if (b.num_records == 0) { stats_ = pairhmm_stats_t{}; return PAIRHMM_OK; }
    if (!b.reads_per_record || !b.haps_per_record) return fail(PAIRHMM_ERR_INVALID_ARGUMENT, "null record arrays");
    if (opts_.gcp && !b.gcp_quals) return fail(PAIRHMM_ERR_INVALID_ARGUMENT, "gcp mode needs the gcp quality array");
    // the host needs the record structure and lengths to derive the index
    std::vector<int32_t> rpr(b.num_records), hpr(b.num_records);
    PHMM_CUDA(cudaMemcpyAsync(rpr.data(), b.reads_per_record, 4 * b.num_records, cudaMemcpyDeviceToHost, stream));
    PHMM_CUDA(cudaMemcpyAsync(hpr.data(), b.haps_per_record, 4 * b.num_records, cudaMemcpyDeviceToHost, stream));
    PHMM_CUDA(cudaStreamSynchronize(stream));
    int64_t nr = 0, nh = 0;
    for (int64_t g = 0; g < b.num_records; ++g) { nr += std::max(rpr[g], 0); nh += std::max(hpr[g], 0); }
    std::vector<int32_t> rl(nr), hl(nh);
    if (nr) PHMM_CUDA(cudaMemcpyAsync(rl.data(), b.read_lengths, 4 * nr, cudaMemcpyDeviceToHost, stream));
    if (nh) PHMM_CUDA(cudaMemcpyAsync(hl.data(), b.hap_lengths, 4 * nh, cudaMemcpyDeviceToHost, stream));
    PHMM_CUDA(cudaStreamSynchronize(stream));
    pairhmm_batch_t hb = b;
    hb.reads_per_record = rpr.data();
    hb.haps_per_record = hpr.data();
    hb.read_lengths = rl.data();
    hb.hap_lengths = hl.data();
    hb.read_offsets = nullptr;
    hb.hap_offsets = nullptr;
    std::string err;
    int64_t pairs = 0;
    for (int64_t g = 0; g < b.num_records; ++g) pairs += (int64_t)std::max(rpr[g], 0) * std::max(hpr[g], 0);
    choose_table(b.num_records, rpr.data(), hpr.data(), rl.data(), pairs);
    pairhmm_status_t st = build_index(hb, table_->rules, *fp64_, idx_, err);
    const BatchIndex& x = idx_;
    if (st != PAIRHMM_OK) return fail(st, err);
    stats_ = pairhmm_stats_t{};
    stats_.pairs = x.num_pairs;
    stats_.cells = x.cells;
    stats_.multi_tile_pairs = x.multi_tile_pairs;
    stats_.rescued = -1;
    stats_.rescued_ext = -1;
    if (x.num_pairs == 0) return PAIRHMM_OK;
    if (!scores) return fail(PAIRHMM_ERR_INVALID_ARGUMENT, "null scores");
    if ((st = ensure_buffers(x)) != PAIRHMM_OK) return st;
    cudaStream_t s = stream_;
    PHMM_CUDA(cudaEventRecord(ev0_, stream));
    PHMM_CUDA(cudaStreamWaitEvent(s, ev0_, 0));
    if ((st = upload_index(x, s)) != PAIRHMM_OK) return st;
    PHMM_CUDA(cudaEventRecord(ev0_, s));
    if ((st = run_pipeline(b, x, scores, s)) != PAIRHMM_OK) return st;
    // an ordinary record behind the graph: the marks are recorded by the graph's nodes
    PHMM_CUDA(cudaEventRecord(fork_, s));
    PHMM_CUDA(cudaStreamWaitEvent(stream, fork_, 0));
    stats_.total_ms = std::chrono::duration<double, std::milli>(std::chrono::steady_clock::now() - t0).count();
    stats_.device_ms = -1.0;
    return PAIRHMM_OK;
}

}  // namespace phmm
