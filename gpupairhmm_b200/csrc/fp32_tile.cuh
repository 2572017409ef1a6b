// __global__ wrapper around the FP32 TileWavefront (wavefront_tile.cuh) and its
// registration.
#pragma once

#include "kernels.hpp"
#include "wavefront_tile.cuh"

namespace phmm {

// Resident blocks per SM asked of the register allocator.  One-warp groups run in
// 64-thread blocks: the paths with per-position w and x hold 8R + ~50 registers a
// lane (packed), so up to R = 10 six blocks fit 168 registers and beyond that four
// blocks (182-255 registers allocated at R = 11-20, the one-gap-quality path's too: both
// paths are one kernel).  The shared tables, 2.5 KB a warp and position pair, are 51 KB a
// block at R = 19-20, where four blocks fit whatever the registers are.  Blocks of 8 warps
// spill 4-60 bytes at R = 8-16.
// Scalar groups hold 4R + ~60: serial parts take eight blocks up to R = 14 and six up
// to R = 24 (168 registers), block groups 16 warps.
template <class V, int R, int W, bool SERIAL>
constexpr int tile_min_ctas() {
    return SERIAL ? (R <= 14 ? 8 : 6) : W > 1 ? 16 / W : (R <= 10 ? 6 : 4);
}

template <class V, int G, int R, int W, bool GCP, bool SERIAL>
__global__ void __launch_bounds__(W == 1 || SERIAL ? kBlockThreads : 32 * W, tile_min_ctas<V, R, W, SERIAL>())
fp32_tile_kernel(DevView v, const Item* __restrict__ items, long long num_items, unsigned long long* counter,
                 void* scratch, int64_t rows) {
    using T = TileWavefront<V, G, R, W, GCP, false, SERIAL>;
    extern __shared__ float4 smem_all[];
    float* ph = reinterpret_cast<float*>(smem_all);  // 128 probabilities
    float4* smem = smem_all + 32;
    for (int i = threadIdx.x; i < 128; i += blockDim.x) ph[i] = v.ph2pr[i];
    __syncthreads();
    constexpr int kWarps = T::kWarps;
    static_assert(T::kBlockGroup || kWarps == kWarpsPerBlock, "independent warps");
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    auto* tab = reinterpret_cast<typename T::Word*>(smem) + warp * T::kTableWords;
    auto* ring = reinterpret_cast<typename T::RingRow*>(reinterpret_cast<char*>(smem) + kWarps * T::kSmemBytes) +
                 (SERIAL ? warp * T::kRing : 0);
    auto* border = SERIAL ? static_cast<typename T::RingRow*>(scratch) +
                                ((int64_t)blockIdx.x * kWarps + warp) * rows
                          : nullptr;
    __shared__ unsigned next;
    const unsigned ntasks = (unsigned)((num_items + T::NG - 1) / T::NG);
    while (true) {
        unsigned x = 0;
        if constexpr (!T::kBlockGroup) {
            if (lane == 0) x = (unsigned)atomicAdd(counter, 1ull);
        } else {
            if (threadIdx.x == 0) next = (unsigned)atomicAdd(counter, 1ull);
            __syncthreads();
            x = next;
            __syncthreads();  // all have it before the next round's write
        }
        // a warp reduction, not a shuffle: the compiler then knows the loop to be
        // uniform and keeps the uniform path's w and x in uniform registers
        x = __reduce_max_sync(kFullMask, x);
        if (x >= ntasks) break;
        const long long first = (long long)x * T::NG;
        const int ntask = (int)min((long long)T::NG, num_items - first);

        const int grp = lane / G;
        const int t = lane - grp * G;
        const bool active = grp < ntask;
        const Item* item = items + first + (active ? grp : 0);
        typename T::Sum sum;
#pragma unroll
        for (int s = 0; s < T::NS; ++s) sum.s[s] = 0.0;
        {
            const Item it = *item;
            const int H = v.hap_len[it.hap];
            const PackedHap hap(reinterpret_cast<const uint32_t*>(v.hap_code + v.hap_start[it.hap]), H);
            typename T::Reads rd;
            unsigned kmin = kNoKey, kmax = 0;
#pragma unroll
            for (int s = 0; s < T::NS; ++s) {
                const int read = s && it.read1 >= 0 ? it.read1 : it.read0;
                rd.L[s] = v.read_len[read];
                rd.read[s].p = v.read_pack + v.read_start[read];
                rd.beta[s] = kBeta;
                rd.inv_beta[s] = 1.0f / kBeta;
                if constexpr (GCP) {
                    rd.eps[s] = ph[v.read_gcp[read]];
                    rd.beta[s] = (float)(1.0 - (double)rd.eps[s]);  // gpuworker.cuh:1049
                    rd.inv_beta[s] = 1.0f / rd.beta[s];
                }
                const unsigned key = v.read_meta[read].key;
                kmin = min(kmin, key);
                kmax = max(kmax, key);
            }
            // every read of the task has the one gap quality
            const bool uni = __reduce_min_sync(kFullMask, kmin) == __reduce_max_sync(kFullMask, kmax) &&
                             kmax != kNoKey;
            const int K = T::kBlockGroup ? 0 : (int)((__reduce_max_sync(kFullMask, (unsigned)(H + G)) + 3u) & ~3u);
            double stop = 0.0;
            if (SERIAL && v.rescue_enabled)
                stop = (double)tile_threshold(rd.L[0], H, v.read_meta[item->read0].range, rd.beta[0]);
            rd.ph = ph;
            T::run(rd, hap, H, K, uni, tab, ring, border, rows, t, T::kBlockGroup ? warp : 0, lane, stop, sum);
        }

        // a serial pair that stopped has no sum: below any threshold
        if (active && t == G - 1 && (!T::kBlockGroup || warp == W - 1)) {
            // the item is read again rather than kept in registers over the steps
            const volatile Item* vi = item;
            const int hap = vi->hap;
            const int H = v.hap_len[hap];
#pragma unroll
            for (int s = 0; s < T::NS; ++s) {
                const int read = s ? vi->read1 : vi->read0;
                if (read < 0) break;
                const int64_t out = s ? vi->out1 : vi->out0;
                const int L = v.read_len[read];
                const ReadMeta meta = v.read_meta[read];
                v.scores[out] = (float)(log10(sum.s[s] / (double)H) - log10((double)kTileD0) - (double)meta.bias);
                const float beta = GCP ? (float)(1.0 - (double)ph[v.read_gcp[read]]) : kBeta;
                if ((meta.flags & 1u) ||
                    (v.rescue_enabled && !(sum.s[s] >= (double)tile_threshold(L, H, meta.range, beta) &&
                                           sum.s[s] <= (double)FLT_MAX)))
                    append_rescue(v, L, Task{read, hap, out});
            }
        }
        __syncwarp();
    }
}

template <class V, int G, int R, int W, bool GCP, bool SERIAL = false>
cudaError_t launch_fp32_tile(const Fp32LaunchArgs& a) {
    using T = TileWavefront<V, G, R, W, GCP, false, SERIAL>;
    fp32_tile_kernel<V, G, R, W, GCP, SERIAL><<<a.grid, 32 * T::kWarps, T::kBlockSmem, a.stream>>>(
        a.view, a.items, a.num_items, a.counter, a.scratch, a.rows);
    return cudaGetLastError();
}

template <class V, int G, int R, int W, bool GCP, bool SERIAL = false>
ConfigInfo make_tile_config() {
    using T = TileWavefront<V, G, R, W, GCP, false, SERIAL>;
    ConfigInfo c{};
    c.G = T::kLanes;
    c.R = R;
    c.multi_tile = W > 1;
    c.packed = T::NS == 2;
    c.exact = true;
    c.gcp = GCP;
    c.per_task = T::NG;
    c.block_threads = 32 * T::kWarps;
    c.tasks_per_block = T::kBlockGroup ? 1 : T::kWarps;
    c.smem_bytes = T::kBlockSmem;
    c.scratch_bytes_per_row = SERIAL ? sizeof(typename T::RingRow) : 0;
    c.kernel = reinterpret_cast<const void*>(&fp32_tile_kernel<V, G, R, W, GCP, SERIAL>);
    c.launch = &launch_fp32_tile<V, G, R, W, GCP, SERIAL>;
    return c;
}

// configurations G x R for R in [R0, R1], packed, both modes
template <int G, int R0, int R1, bool GCP>
void register_tiles(std::vector<ConfigInfo>& out) {
    if constexpr (R0 <= R1) {
        out.push_back(make_tile_config<float2, G, R0, 1, GCP>());
        register_tiles<G, R0 + 1, R1, GCP>(out);
    }
}

// configurations of 32*W lanes x R, one read per group: blocks of W warps, or one warp
// with W parts in turn
template <int W, int R0, int R1, bool GCP, bool SERIAL>
void register_long(std::vector<ConfigInfo>& out) {
    if constexpr (R0 <= R1) {
        out.push_back(make_tile_config<float, 32, R0, W, GCP, SERIAL>());
        register_long<W, R0 + 1, R1, GCP, SERIAL>(out);
    }
}

}  // namespace phmm
