// __global__ wrapper around the FP32 TileWavefront (wavefront_tile.cuh) and its
// registration.
#pragma once

#include "kernels.hpp"
#include "wavefront_tile.cuh"

namespace phmm {

// Resident blocks per SM asked of the register allocator.  One-warp groups run in
// 64-thread blocks: the paths with per-position w and x hold 8R + ~50 registers a
// lane (packed), so up to R = 10 six blocks fit 168 registers and beyond that four
// blocks; the shared tables (2.5 KB a warp and position pair) allow as many.
template <class V, int R, int W>
constexpr int tile_min_ctas() {
    return W > 1 ? 16 / W : (R <= 10 ? 6 : 4);
}

template <class V, int G, int R, int W, bool GCP>
__global__ void __launch_bounds__(W == 1 ? kBlockThreads : 32 * W, tile_min_ctas<V, R, W>())
fp32_tile_kernel(DevView v, const Item* __restrict__ items, long long num_items, unsigned long long* counter) {
    using T = TileWavefront<V, G, R, W, GCP>;
    extern __shared__ float4 smem[];
    constexpr int kWarps = W == 1 ? kWarpsPerBlock : W;
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    auto* tab = reinterpret_cast<typename T::Word*>(smem) + warp * T::kTableWords;
    auto* ring = reinterpret_cast<typename T::RingRow*>(reinterpret_cast<char*>(smem) + kWarps * T::kSmemBytes);
    __shared__ unsigned next;
    const unsigned ntasks = (unsigned)((num_items + T::NG - 1) / T::NG);
    while (true) {
        unsigned x = 0;
        if constexpr (W == 1) {
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
        double acc[T::NS];
#pragma unroll
        for (int s = 0; s < T::NS; ++s) acc[s] = 0.0;
        {
            const Item it = *item;
            const int H = v.hap_len[it.hap];
            const uint32_t* hw = reinterpret_cast<const uint32_t*>(v.hap_code + v.hap_start[it.hap]);
            typename T::Reads rd;
            unsigned kmin = kNoKey, kmax = 0;
#pragma unroll
            for (int s = 0; s < T::NS; ++s) {
                const int read = s && it.read1 >= 0 ? it.read1 : it.read0;
                rd.L[s] = v.read_len[read];
                const int64_t start = v.read_start[read];
                rd.coef[s] = v.read_coef + start;
                rd.pack[s] = v.read_pack + start;
                rd.w_end[s] = v.read_meta[read].w_end;
                if constexpr (GCP) rd.eps[s] = v.ph2pr[v.read_gcp[read]];
                const unsigned key = v.read_meta[read].key;
                kmin = min(kmin, key);
                kmax = max(kmax, key);
            }
            // every read of the task has the one gap quality
            const bool uni = __reduce_min_sync(kFullMask, kmin) == __reduce_max_sync(kFullMask, kmax) &&
                             kmax != kNoKey;
            const int K = W == 1 ? (int)((__reduce_max_sync(kFullMask, (unsigned)(H + G)) + 3u) & ~3u) : 0;
            if (uni) T::template loop<true>(rd, hw, H, K, tab, ring, t, W == 1 ? 0 : warp, lane, acc);
            else T::template loop<false>(rd, hw, H, K, tab, ring, t, W == 1 ? 0 : warp, lane, acc);
        }

        if (active && t == G - 1 && (W == 1 || warp == W - 1)) {
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
                v.scores[out] = (float)(log10(acc[s] / (double)H) - log10((double)kTileD0));
                if ((meta.flags & 1u) ||
                    (v.rescue_enabled && !(acc[s] >= (double)tile_threshold(L, H, meta.range) &&
                                           acc[s] <= (double)FLT_MAX)))
                    append_rescue(v, fp64_class(L), Task{read, hap, out});
            }
        }
        __syncwarp();
    }
}

template <class V, int G, int R, int W, bool GCP>
cudaError_t launch_fp32_tile(const Fp32LaunchArgs& a) {
    using T = TileWavefront<V, G, R, W, GCP>;
    constexpr int kWarps = W == 1 ? kWarpsPerBlock : W;
    fp32_tile_kernel<V, G, R, W, GCP><<<a.grid, 32 * kWarps, kWarps * T::kSmemBytes + T::kRingBytes, a.stream>>>(
        a.view, a.items, a.num_items, a.counter);
    return cudaGetLastError();
}

template <class V, int G, int R, int W, bool GCP>
ConfigInfo make_tile_config() {
    using T = TileWavefront<V, G, R, W, GCP>;
    constexpr int kWarps = W == 1 ? kWarpsPerBlock : W;
    ConfigInfo c{};
    c.G = T::NL;
    c.R = R;
    c.multi_tile = W > 1;
    c.packed = T::NS == 2;
    c.exact = true;
    c.gcp = GCP;
    c.per_task = T::NG;
    c.block_threads = 32 * kWarps;
    c.tasks_per_block = W == 1 ? kWarpsPerBlock : 1;
    c.smem_bytes = kWarps * T::kSmemBytes + T::kRingBytes;
    c.kernel = reinterpret_cast<const void*>(&fp32_tile_kernel<V, G, R, W, GCP>);
    c.launch = &launch_fp32_tile<V, G, R, W, GCP>;
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

}  // namespace phmm
