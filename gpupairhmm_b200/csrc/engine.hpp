// Host-side engine behind the C ABI.
#pragma once

#include <cuda_runtime.h>

#include <cstdint>
#include <memory>
#include <string>
#include <unordered_map>
#include <vector>

#include "../../include/pairhmm_b200.h"
#include "host_upload.hpp"
#include "kernels.hpp"

namespace phmm {

// One entry of a tile table: reads with length <= max_len (and above the
// previous entry's bound) run with (G, R, multi_tile).
struct TileRule {
    int max_len;
    int G;
    int R;
    bool multi_tile;
    bool packed = false;  // two reads of a record per group, packed FP32
    bool exact = false;   // lanes hold R or R-1 positions (wavefront_tile.cuh)
};

inline bool operator==(const TileRule& a, const TileRule& b) {
    return a.max_len == b.max_len && a.G == b.G && a.R == b.R && a.multi_tile == b.multi_tile &&
           a.packed == b.packed && a.exact == b.exact;
}

// A tile table with its compiled kernels.
struct TileTable {
    std::vector<TileRule> rules;
    std::vector<const ConfigInfo*> cfg;
};

// Length classes of the FP64 pass and their kernels.
struct Fp64Table {
    struct Class {
        int max_len;
        const Fp64Config* scaled;
        int ext;                      // extended-tier class of its pairs
    };
    struct Ext {
        const Fp64Config* cfg;
        int first, last;              // its scaled classes
        bool own_stream;              // one scaled class: runs right behind it
    };
    std::vector<Class> classes;
    std::vector<Ext> exts;
    const Fp64Config* fused = nullptr;  // fused form of the last class
    std::vector<uint8_t> lut;           // class of a read length (kFp64LutSize)
    int class_of(int L) const { return lut.empty() ? 0 : lut[L <= kFp64LutMax ? L : kFp64LutMax + 1]; }
};

// Per-batch index derived on the host from the record structure.
struct BatchIndex {
    int64_t num_records = 0, num_reads = 0, num_haps = 0, num_pairs = 0, cells = 0;
    int32_t max_read_len = 0, max_hap_len = 0;
    int64_t read_bytes = 0, hap_bytes = 0;          // end of the caller's referenced byte range
    int64_t read_min = 0, hap_min = 0;              // start of that range
    int64_t pack_positions = 0, code_bytes = 0;     // packed extents
    std::vector<int32_t> read_record, read_local, rec_haps;
    std::vector<int64_t> rec_hap_base, rec_pair_base, read_start, hap_start;
    std::vector<int64_t> bucket_pairs;              // by bucket index
    std::vector<int64_t> bucket_items;              // work items (unit x haplotype) by bucket
    std::vector<int32_t> unit_read0, unit_read1, unit_bucket;  // units: 1 or 2 reads of a record
    int64_t class_pairs[kMaxFp64Classes] = {};      // by FP64 length class
    // starts of the FP64 lists: the scaled tier's by class, then the extended tier's by
    // its classes (each holds the pairs of consecutive scaled classes)
    int64_t list_start[2 * kMaxFp64Classes] = {};
    int64_t multi_tile_pairs = 0;
};

// Sizes and referenced byte ranges of a host batch, validated (first pass,
// cheap: lets the input upload start before the index is built).
struct InputRanges {
    int64_t num_reads = 0, num_haps = 0, num_pairs = 0;
    int64_t read_min = 0, read_end = 0, hap_min = 0, hap_end = 0;
};

// Grow-only device buffer.  With a pool and a stream set (every engine
// buffer), growth is stream-ordered (cudaFreeAsync + cudaMallocFromPoolAsync
// on the engine's stream): unlike cudaFree it does not wait for the whole
// device, so one engine growing its buffers does not stall other engines'
// work (serving runs several).
struct DevBuf {
    void* ptr = nullptr;
    size_t cap = 0;
    cudaMemPool_t pool = nullptr;
    cudaStream_t stream = nullptr;
    cudaError_t ensure(size_t bytes);
    void release();
    template <class T> T* as() const { return static_cast<T*>(ptr); }
};

class Engine {
public:
    explicit Engine(const pairhmm_options_t& opts);
    ~Engine();
    Engine(const Engine&) = delete;
    Engine& operator=(const Engine&) = delete;

    // The host thread waits for what a launch depends on, instead of enqueueing the launch
    // with a wait ahead of it.  A device has 8 launch queues (by default), which all streams
    // share in turn, and a wait in one holds up every later launch in it, whichever stream
    // that is of: for engines with long kernels beside ones with short batches (serving.cu).
    void set_staged(bool on) { staged_ = on; }
    pairhmm_status_t init();
    // keeps `bytes` of device memory in the engine's pool (allocated once and freed), so
    // that buffer growth up to that size maps no new memory while other work runs
    pairhmm_status_t reserve_pool(size_t bytes);
    // loads every kernel of the engine's tables and makes its side streams, so that no batch's
    // first use of a class does
    pairhmm_status_t load_all();
    pairhmm_status_t compute_host(const pairhmm_batch_t& b, float* scores);
    pairhmm_status_t compute_device(const pairhmm_batch_t& b, int32_t max_read_len, int32_t max_hap_len,
                                    float* scores, cudaStream_t stream);
    const pairhmm_stats_t& stats() const { return stats_; }
    const std::string& last_error() const { return last_error_; }
    pairhmm_status_t fail(pairhmm_status_t s, const std::string& msg);
    pairhmm_status_t cuda_fail(cudaError_t e, const char* what);

    // Replace the tile table of the current mode (autotuner).
    pairhmm_status_t set_tile_table(const std::vector<TileRule>& rules);
    const std::vector<TileRule>& tile_table() const { return tables_[0].rules; }
    // engine form with the table it was made with
    bool has_default_table() const { return has_default_table(tables_[0].rules); }
    int device() const { return opts_.device; }
    bool gcp() const { return opts_.gcp != 0; }
    int64_t budget_bytes() const { return opts_.device_budget_bytes; }
    int num_sms() const { return num_sms_; }

    static pairhmm_status_t build_index(const pairhmm_batch_t& b, const std::vector<TileRule>& rules,
                                        const Fp64Table& fp64, BatchIndex& idx, std::string& err);
    // gcp: the batch must carry gcp qualities, none 0 at a read's first position
    static pairhmm_status_t scan_inputs(const pairhmm_batch_t& b, InputRanges& r, std::string& err, bool gcp);

private:
    // compute_host in two halves: everything enqueued / the wait and results
    pairhmm_status_t host_begin(const pairhmm_batch_t& b, float* scores, cudaEvent_t mark_start,
                                cudaEvent_t mark_end);
    pairhmm_status_t host_end();
    bool has_default_table(const std::vector<TileRule>& rules) const;
    pairhmm_status_t build_tables(const std::vector<TileRule>& rules);
    // the table for a batch of these records becomes the current one
    void choose_table(int64_t num_records, const int32_t* reads_per_record, const int32_t* haps_per_record,
                      const int32_t* read_lengths, int64_t pairs);
    pairhmm_status_t run_pipeline(const pairhmm_batch_t& dev_in, const BatchIndex& idx, float* d_scores,
                                  cudaStream_t s);
    struct Plan {
        int64_t rows = 0;                 // border rows per buffer
        std::vector<int> grid;            // by bucket
        std::vector<int> persistent;      // by bucket
        int fp64_grid[kMaxFp64Classes] = {};      // by FP64 length class: scaled tier
        int fp64_ext_grid[kMaxFp64Classes] = {};  // by extended-tier class
        int64_t fp64_scratch[kMaxFp64Classes] = {};      // border scratch offsets of the
        int64_t fp64_ext_scratch[kMaxFp64Classes] = {};  // kernels that need it
        int side[3] = {};                 // side streams of a stage: one per launch, up to kSideStreams
        std::vector<int64_t> scratch_off;   // by bucket: multi-tile kernels run side by side
        size_t scratch_bytes = 0;
    };
    Plan make_plan(const BatchIndex& idx) const;
    int64_t fp64_warps(const BatchIndex& x) const;
    std::vector<uint8_t> launch_shape(const BatchIndex& x, const Plan& plan) const;
    // stage 0: packing + work list, 1: FP32 launches, 2: FP64 pass
    pairhmm_status_t enqueue_pipeline(const pairhmm_batch_t& dev_in, const BatchIndex& idx, const Plan& plan,
                                      float* d_scores, cudaStream_t s, int stage);
    pairhmm_status_t ensure_buffers(const BatchIndex& idx);
    pairhmm_status_t ensure_inputs(const InputRanges& r);
    // The index (and, gathered, the inputs too: `in` points at the host arrays and comes
    // back pointing at device copies) onto the device.
    pairhmm_status_t upload_index(const BatchIndex& idx, cudaStream_t s);
    pairhmm_status_t upload_gathered(const BatchIndex& idx, const InputRanges* r, pairhmm_batch_t* in,
                                     cudaStream_t s);
    static size_t input_bytes(const InputRanges& r, bool gcp);
    pairhmm_status_t load_kernels(const TileTable& table, const Fp64Table& fp64, const BatchIndex* x);
    pairhmm_status_t load_kernel(const void* kernel, int threads, size_t smem);
    int persistent_grid(const void* kernel) const;
    static int64_t index_bytes(const BatchIndex& x);
    int64_t hbins_of(const BatchIndex& x) const;

    pairhmm_options_t opts_;
    // tables_[0] is the engine's table, tables_[1] (default tables only) the one for
    // batches of few pairs, with groups as wide as possible (choose_table)
    TileTable tables_[2];
    const TileTable* table_ = &tables_[0];
    Fp64Table fp64_tables_[2];          // FP64 classes: on 8-32 lanes, and as wide as possible
    const Fp64Table* fp64_ = &fp64_tables_[0];
    DevBuf fp64_lut_[2];
    int num_sms_ = 0;
    std::unordered_map<const void*, int> blocks_per_sm_;  // kernels loaded so far
    bool ready_ = false;
    cudaStream_t stream_ = nullptr;
    // the launches of one stage (bucket kernels, FP64 classes) fork onto side
    // streams so that their tails overlap and a small batch's buckets run side
    // by side; they join back into stream_ before the stage ends
    static constexpr int kSideStreams = 16;
    bool staged_ = false;
    cudaStream_t side_[kSideStreams] = {};   // created as batches need them
    cudaEvent_t fork_ = nullptr, join_[kSideStreams] = {};
    pairhmm_status_t ensure_side_streams(int n);
    cudaEvent_t ev0_ = nullptr, ev1_ = nullptr, ev_prep_ = nullptr, ev_fp32_ = nullptr;
    int64_t launches_ = 0, fp32_launches_ = 0;
    cudaGraphExec_t graph_exec_ = nullptr;   // the whole batch: prep, FP32, FP64
    std::vector<uint8_t> graph_shape_, last_shape_;  // launch_shape of the kept graph and of the last batch
    int64_t shape_repeats_ = 0;               // batches before the last one with its shape, in a row
    pairhmm_stats_t stats_{};
    std::string last_error_;

    // device buffers
    DevBuf ph2pr_;
    DevBuf in_read_bases_, in_bq_, in_iq_, in_dq_, in_read_off_, in_read_len_;
    DevBuf in_gq_, read_gcp_;  // gcp mode: uploaded gcp qualities, per-read gcp
    DevBuf in_hap_bases_, in_hap_off_, in_hap_len_;
    DevBuf read_record_, read_local_, rec_haps_, rec_hap_base_, rec_pair_base_, read_start_, hap_start_;
    DevBuf unit_read0_, unit_read1_, unit_bucket_;
    DevBuf arena_;   // a small batch's inputs and index, uploaded in one copy
    // the current batch's index on the device
    struct IndexPtrs {
        const int32_t *read_record, *read_local, *rec_haps, *unit_read0, *unit_read1, *unit_bucket;
        const int64_t *rec_hap_base, *rec_pair_base, *read_start, *hap_start;
        const long long* list_start;
    } ix_{};
    DevBuf read_pack_, read_meta_, hap_code_, hist_, cursor_, items_, rescue_, counters_, scores_, scratch_;
    DevBuf rescue_off_, rescue_ext_, rsort_;
    // host-to-device uploads (caller inputs, index) and the reused index
    HostUploader uploader_;
    BatchIndex idx_;
    // pipelined compute_host: chunks of at least kChunkPairs pairs (up to
    // kMaxChunks) alternate between this engine and its twin; only the first
    // chunk's upload is exposed (uneven workload, 10.9 M pairs: 8 chunks 185.1 ms,
    // 4 chunks 186.8 ms end to end)
    // pairs per occupied length class up to which a batch counts as small
    static constexpr int64_t kSmallPairs = 1024;
    static constexpr int64_t kChunkPairs = int64_t(1) << 20;
    static constexpr int64_t kMaxChunks = 8;
    std::unique_ptr<Engine> twin_;
    cudaEvent_t span0_ = nullptr, span1_ = nullptr;
    bool pending_ = false, pend_direct_ = false;
    float* pend_scores_ = nullptr;
    int64_t pend_pairs_ = 0;
    // page-locked landing spot for the rescue counts (both FP64 tiers)
    void* host_hdr_ = nullptr;
    // device memory pool of this engine's buffers (kept, not returned to the
    // system between batches)
    cudaMemPool_t pool_ = nullptr;
    std::vector<DevBuf*> all_buffers();
};

}  // namespace phmm
