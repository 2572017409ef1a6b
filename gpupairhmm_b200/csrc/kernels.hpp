// Host-visible registry of the compiled kernel configurations.
#pragma once

#include <cuda_runtime.h>

#include <cstddef>
#include <cstdint>
#include <vector>

#include "device_common.cuh"
#include "prep_kernels.cuh"

namespace phmm {

constexpr int kBlockThreads = 64;  // 2 warps per CTA: register-bound configs reach 10 warps/SM
constexpr int kWarpsPerBlock = kBlockThreads / 32;

struct Fp32LaunchArgs {
    DevView view;
    const Item* items;              // the bucket's first work item
    long long num_items;
    int persistent;                 // 1: warps loop on an atomic task counter
    unsigned long long* counter;    // per-rank task counter (persistent)
    void* scratch;                  // multi-tile border storage
    int64_t rows;                   // border rows per buffer
    int grid;
    cudaStream_t stream;
};

struct Fp64LaunchArgs {
    DevView view;
    ExtList ext_list;                // scaled tier: where pairs beyond its range go
    const Task* items;               // the class's rescue list
    const unsigned long long* count; // number of items (device)
    unsigned long long* counter;     // task counter
    void* scratch;                   // border storage (padded multi-tile kernels only)
    int64_t rows;
    int grid;
    cudaStream_t stream;
};

// A compiled kernel of the FP64 pass.  Exact tiles take reads of (G*(R-1), G*R]
// positions; the padded kernels (wavefront_fp64.cuh) up to G*R, or any length
// (multi_tile).
struct Fp64Config {
    int G;
    int R;
    bool ext;                        // extended tier (per-lane exponents)
    bool gcp;
    bool exact;
    bool multi_tile;                 // padded kernel, tile after tile
    bool fused;                      // scaled tier that runs a pair's extended form in the same warp
    int per_task;
    int block_threads;
    int tasks_per_block;
    size_t smem_bytes;
    size_t scratch_bytes_per_row;    // per warp, per border row
    const void* kernel;
    cudaError_t (*launch)(const Fp64LaunchArgs&);
};

struct ConfigInfo {
    int G;                           // lanes per group (above 32: the warps of a block)
    int R;
    bool multi_tile;                 // reads beyond one warp's tile
    bool packed;                     // two reads per group with packed FP32
    bool exact;                      // wavefront_tile.cuh: read lengths (G*(R-1), G*R] only
    bool gcp;                        // eps/beta per read (gcp mode)
    int per_task;                    // items per task (of a warp, or of a block)
    int block_threads;
    int tasks_per_block;             // tasks a block works on at a time
    size_t smem_bytes;               // dynamic shared memory per CTA
    size_t scratch_bytes_per_row;    // per warp, per border row (both buffers)
    const void* kernel;
    cudaError_t (*launch)(const Fp32LaunchArgs&);
};

// All compiled FP32 configurations.
const std::vector<ConfigInfo>& fp32_configs();
const ConfigInfo* find_fp32_config(int G, int R, bool multi_tile, bool packed, bool exact, bool gcp);

// All compiled kernels of the FP64 pass.  The scaled tier (ext = false) recomputes
// every flagged pair, the extended tier (ext = true) the pairs beyond its range.
const std::vector<Fp64Config>& fp64_configs();
const Fp64Config* find_fp64_config(int G, int R, bool exact, bool ext, bool gcp, bool fused = false);

// Preparation kernels.  The pack launch also runs the batch's fills.
cudaError_t launch_pack(const PrepArgs& a, const FillArgs& f, int grid, cudaStream_t s);
// FP64 class lists sorted by haplotype length (count, scan, scatter)
cudaError_t launch_rescue_sort(const RescueSortArgs& a, int grid, cudaStream_t s);
cudaError_t launch_binning(const BinArgs& a, int grid, cudaStream_t s);

// FP32 FFMA throughput probe used to measure the roofline denominator:
// `iters` dependent-chain-free FMAs per thread over grid x 256 threads.
cudaError_t launch_ffma_peak(float* out, int grid, int iters, cudaStream_t s);
// The same with double FMAs.
cudaError_t launch_dfma_peak(float* out, int grid, int iters, cudaStream_t s);

}  // namespace phmm
