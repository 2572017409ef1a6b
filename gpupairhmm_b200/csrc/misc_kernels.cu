// FP64 rescue kernel, preparation launchers, configuration registry and the
// FFMA throughput probe.
#include <algorithm>
#include <mutex>

#define PHMM_PREP_KERNELS_IMPL
#include "kernels.hpp"
#include "prep_kernels.cuh"
#include "wavefront_fp64.cuh"

namespace phmm {

void register_fp32_g4(std::vector<ConfigInfo>& out);
void register_fp32_g8(std::vector<ConfigInfo>& out);
void register_fp32_g16(std::vector<ConfigInfo>& out);
void register_fp32_g32(std::vector<ConfigInfo>& out);
void register_fp32_gcp(std::vector<ConfigInfo>& out);
void register_fp32_geven(std::vector<ConfigInfo>& out);
void register_tile_g8(std::vector<ConfigInfo>& out);
void register_tile_g16(std::vector<ConfigInfo>& out);
void register_tile_g32(std::vector<ConfigInfo>& out);
void register_tile_gcp_g8(std::vector<ConfigInfo>& out);
void register_tile_gcp_g16(std::vector<ConfigInfo>& out);
void register_tile_gcp_g32(std::vector<ConfigInfo>& out);
void register_long(std::vector<ConfigInfo>& out);
void register_long_gcp(std::vector<ConfigInfo>& out);

const std::vector<ConfigInfo>& fp32_configs() {
    static std::vector<ConfigInfo> all;
    static std::once_flag once;
    std::call_once(once, [] {
        register_fp32_g4(all);
        register_fp32_g8(all);
        register_fp32_g16(all);
        register_fp32_g32(all);
        register_fp32_geven(all);
        register_fp32_gcp(all);
        register_tile_g8(all);
        register_tile_g16(all);
        register_tile_g32(all);
        register_tile_gcp_g8(all);
        register_tile_gcp_g16(all);
        register_tile_gcp_g32(all);
        register_long(all);
        register_long_gcp(all);
    });
    return all;
}

const ConfigInfo* find_fp32_config(int G, int R, bool multi_tile, bool packed, bool exact, bool gcp) {
    for (const auto& c : fp32_configs())
        if (c.G == G && c.R == R && c.exact == exact && (exact || c.multi_tile == multi_tile) && c.packed == packed &&
            c.gcp == gcp)
            return &c;
    return nullptr;
}

// ---------------------------------------------------------------- FP64 pass
// Padded kernels of the FP64 pass (wavefront_fp64.cuh), where fp64_tile.cuh has no
// exact tile: both tiers of reads up to 32 positions and beyond 4,096, and the
// extended tier of reads up to 640, which few pairs reach.  A step's cost is mostly
// per lane (hand-off, scale conversion, renormalisation), so the tiles take 12-16
// positions per lane where the registers allow; 160 keeps 16 x 10 at 168 registers.
template <bool EXT> using W64c0 = Fp64Wavefront<4, 16, false, false, EXT>;
template <bool EXT> using W64c1 = Fp64Wavefront<8, 12, false, false, EXT>;
template <bool EXT> using W64c2 = Fp64Wavefront<8, 16, false, false, EXT>;
template <bool EXT> using W64c3 = Fp64Wavefront<16, 10, false, false, EXT>;
template <bool EXT> using W64c4 = Fp64Wavefront<16, 12, false, false, EXT>;
template <bool EXT> using W64c5 = Fp64Wavefront<16, 16, false, false, EXT>;
template <bool EXT> using W64c6 = Fp64Wavefront<32, 16, true, false, EXT>;

// The multi-tile kernel's scaled tier runs the extended form of a pair right after
// it in the same warp when the pair needs it (FUSE), so the border ring and the
// scratch rows are sized for the extended form's 32-byte rows.
template <class W>
using Fp64ExtOf = Fp64Wavefront<W::G_, W::R_, W::kMT, W::kGCP, true>;
template <class W>
constexpr size_t fp64_ring_entry() { return W::kMT ? sizeof(Border64) : sizeof(typename W::Border); }

// FUSE (multi-tile scaled tier): a pair that needs the extended tier runs it
// right away in the same warp, instead of waiting in the extended tier's list
// for a launch of its own; for batches of a few long regions (one long pair is
// a long serial wavefront) that takes the second pass off their latency.
template <class W, bool FUSE>
__global__ void __launch_bounds__(kBlockThreads, W::kMinCtas)
fp64_rescue_kernel(DevView v, const Task* __restrict__ items, const unsigned long long* count,
                   unsigned long long* counter, void* scratch, int64_t rows, ExtList ext) {
    using Border = typename W::Border;
    extern __shared__ double2 smem64[];
    float* ph = reinterpret_cast<float*>(smem64);  // 128 floats = 32 double2
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    double2* wtab = smem64 + 32 + warp * W::kTableDouble2;
    char* ring_bytes = reinterpret_cast<char*>(smem64 + 32 + kWarpsPerBlock * W::kTableDouble2) +
                       (size_t)warp * W::kRing * fp64_ring_entry<W>();
    for (int i = threadIdx.x; i < 128; i += blockDim.x) ph[i] = v.ph2pr[i];
    __syncthreads();
    const unsigned long long n = *count;
    const unsigned long long ntasks = (n + W::NG - 1) / W::NG;
    const long long gwarp = (long long)blockIdx.x * kWarpsPerBlock + warp;
    char* wscratch = scratch ? static_cast<char*>(scratch) + (size_t)gwarp * rows * fp64_ring_entry<W>() : nullptr;
    while (true) {
        unsigned long long x = 0;
        if (lane == 0) x = atomicAdd(counter, 1ull);
        x = __shfl_sync(kFullMask, x, 0);
        if (x >= ntasks) break;
        const unsigned long long first = x * W::NG;
        const int ntask = (int)((n - first) < (unsigned long long)W::NG ? (n - first) : W::NG);
        const bool to_ext = W::run(v, items + first, ntask, ph, wtab, reinterpret_cast<Border*>(ring_bytes),
                                   reinterpret_cast<Border*>(wscratch), rows, ext, FUSE);
        if constexpr (FUSE) {
            if (to_ext) {  // warp-uniform: one pair per warp
                using WE = Fp64ExtOf<W>;
                __syncwarp();
                WE::run(v, items + first, ntask, ph, wtab, reinterpret_cast<typename WE::Border*>(ring_bytes),
                        reinterpret_cast<typename WE::Border*>(wscratch), rows, ext, false);
                if (lane == 0) atomicAdd(ext.count + ext.cls, 1ull);  // counted with the extended tier
            }
        }
    }
}

template <class W>
size_t fp64_smem_for() {
    return (32 + (size_t)kWarpsPerBlock * W::kTableDouble2) * sizeof(double2) +
           (size_t)kWarpsPerBlock * W::kRing * fp64_ring_entry<W>();
}

// gcp-mode twins (same tiles, eps/beta per read)
template <class W>
struct WithGcp;
template <int G, int R, bool MT, bool EXT>
struct WithGcp<Fp64Wavefront<G, R, MT, false, EXT>> {
    using type = Fp64Wavefront<G, R, MT, true, EXT>;
};

template <class W, bool FUSE>
cudaError_t launch_fp64_padded(const Fp64LaunchArgs& a) {
    fp64_rescue_kernel<W, FUSE><<<a.grid, kBlockThreads, fp64_smem_for<W>(), a.stream>>>(
        a.view, a.items, a.count, a.counter, W::kMT ? a.scratch : nullptr, a.rows, a.ext_list);
    return cudaGetLastError();
}

template <class W, bool FUSE = false>
Fp64Config make_padded64_config() {
    Fp64Config c{};
    c.G = W::G_;
    c.R = W::R_;
    c.ext = W::kEXT;
    c.gcp = W::kGCP;
    c.multi_tile = W::kMT;
    c.fused = FUSE;
    c.per_task = W::NG;
    c.block_threads = kBlockThreads;
    c.tasks_per_block = kWarpsPerBlock;
    c.smem_bytes = fp64_smem_for<W>();
    // one border buffer per warp, shared by all tile boundaries of its pair
    c.scratch_bytes_per_row = W::kMT ? sizeof(Border64) : 0;
    c.kernel = reinterpret_cast<const void*>(&fp64_rescue_kernel<W, FUSE>);
    c.launch = &launch_fp64_padded<W, FUSE>;
    return c;
}

template <class W>
void register_padded64(std::vector<Fp64Config>& out) {
    out.push_back(make_padded64_config<W>());
    out.push_back(make_padded64_config<typename WithGcp<W>::type>());
}

void register_tile64_g8(std::vector<Fp64Config>& out);
void register_tile64_g16(std::vector<Fp64Config>& out);
void register_tile64_g32(std::vector<Fp64Config>& out);
void register_long64(std::vector<Fp64Config>& out);
void register_long64_gcp(std::vector<Fp64Config>& out);

const std::vector<Fp64Config>& fp64_configs() {
    static std::vector<Fp64Config> all;
    static std::once_flag once;
    std::call_once(once, [] {
        register_padded64<W64c0<false>>(all);
        register_padded64<W64c6<false>>(all);
        all.push_back(make_padded64_config<W64c6<false>, true>());
        all.push_back(make_padded64_config<WithGcp<W64c6<false>>::type, true>());
        register_padded64<W64c0<true>>(all);
        register_padded64<W64c1<true>>(all);
        register_padded64<W64c2<true>>(all);
        register_padded64<W64c3<true>>(all);
        register_padded64<W64c4<true>>(all);
        register_padded64<W64c5<true>>(all);
        register_padded64<W64c6<true>>(all);
        register_tile64_g8(all);
        register_tile64_g16(all);
        register_tile64_g32(all);
        register_long64(all);
        register_long64_gcp(all);
    });
    return all;
}

const Fp64Config* find_fp64_config(int G, int R, bool exact, bool ext, bool gcp, bool fused) {
    for (const auto& c : fp64_configs())
        if (c.G == G && c.R == R && c.exact == exact && c.ext == ext && c.gcp == gcp && c.fused == fused) return &c;
    return nullptr;
}

// ---------------------------------------------------------------- preparation
cudaError_t launch_pack(const PrepArgs& a, const FillArgs& f, int grid, cudaStream_t s) {
    // a warp per read / haplotype with every warp resident at once where the batch
    // allows: each warp's work is short, so latency is hidden by warps in flight
    auto warps_grid = [&](int64_t n) {
        const int64_t g = (n + 7) / 8;  // 8 warps per 256-thread block
        return (int)std::max<int64_t>(1, std::min<int64_t>(g, int64_t(1) << 20));
    };
    long long most = 0;
    for (long long w : f.words) most = std::max(most, w);
    const int fill_blocks = (int)std::max<long long>(1, std::min<long long>((most + 1023) / 1024, grid));
    const int read_blocks = warps_grid(a.num_reads), hap_blocks = warps_grid(a.num_haps);
    pack_kernel<<<fill_blocks + read_blocks + hap_blocks, 256, 0, s>>>(a, f, fill_blocks, read_blocks);
    return cudaGetLastError();
}

cudaError_t launch_rescue_sort(const RescueSortArgs& a, int grid, cudaStream_t s) {
    rescue_count_kernel<<<grid, 256, 0, s>>>(a);
    rescue_scan_kernel<<<a.classes, 32, 0, s>>>(a);
    rescue_scatter_kernel<<<grid, 256, 0, s>>>(a);
    return cudaGetLastError();
}

cudaError_t launch_binning(const BinArgs& a, int grid, cudaStream_t s) {
    const int units_grid = (int)std::max<int64_t>(1, std::min<int64_t>((a.num_units + 255) / 256, grid));
    bin_count_kernel<<<units_grid, 256, 0, s>>>(a);
    hist_scan_kernel<<<a.nbuckets, kHistScanThreads, 0, s>>>(a.hist, a.cursor, a.hbins, a.ranks);
    bin_scatter_kernel<<<units_grid, 256, 0, s>>>(a);
    return cudaGetLastError();
}

// ---------------------------------------------------------------- FFMA probe
// 8 independent FMA chains per thread; 2 FLOP per FMA.
__global__ void __launch_bounds__(256) ffma_peak_kernel(float* out, int iters) {
    float a0 = threadIdx.x * 1e-3f, a1 = a0 + 1.f, a2 = a0 + 2.f, a3 = a0 + 3.f;
    float a4 = a0 + 4.f, a5 = a0 + 5.f, a6 = a0 + 6.f, a7 = a0 + 7.f;
    const float b = 0.9999f, c = 1e-7f;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            a0 = fmaf(a0, b, c); a1 = fmaf(a1, b, c); a2 = fmaf(a2, b, c); a3 = fmaf(a3, b, c);
            a4 = fmaf(a4, b, c); a5 = fmaf(a5, b, c); a6 = fmaf(a6, b, c); a7 = fmaf(a7, b, c);
        }
    }
    const float s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s == 12345.678f) out[0] = s;  // keeps the chains live
}

cudaError_t launch_ffma_peak(float* out, int grid, int iters, cudaStream_t s) {
    ffma_peak_kernel<<<grid, 256, 0, s>>>(out, iters);
    return cudaGetLastError();
}

// The same with double FMAs (the FP64 pass's roofline denominator).
__global__ void __launch_bounds__(256) dfma_peak_kernel(float* out, int iters) {
    double a0 = threadIdx.x * 1e-3, a1 = a0 + 1.0, a2 = a0 + 2.0, a3 = a0 + 3.0;
    double a4 = a0 + 4.0, a5 = a0 + 5.0, a6 = a0 + 6.0, a7 = a0 + 7.0;
    const double b = 0.9999, c = 1e-7;
    for (int i = 0; i < iters; ++i) {
#pragma unroll
        for (int u = 0; u < 16; ++u) {
            a0 = fma(a0, b, c); a1 = fma(a1, b, c); a2 = fma(a2, b, c); a3 = fma(a3, b, c);
            a4 = fma(a4, b, c); a5 = fma(a5, b, c); a6 = fma(a6, b, c); a7 = fma(a7, b, c);
        }
    }
    const double s = a0 + a1 + a2 + a3 + a4 + a5 + a6 + a7;
    if (s == 12345.678) out[0] = (float)s;  // keeps the chains live
}

cudaError_t launch_dfma_peak(float* out, int grid, int iters, cudaStream_t s) {
    dfma_peak_kernel<<<grid, 256, 0, s>>>(out, iters);
    return cudaGetLastError();
}

}  // namespace phmm
