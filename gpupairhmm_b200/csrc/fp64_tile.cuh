// __global__ wrapper around the FP64 TileWavefront (wavefront_tile.cuh) and its
// registration: the scaled tier's exact tiles, and for groups of several warps the
// extended tier's too.
#pragma once

#include "kernels.hpp"
#include "wavefront_tile.cuh"

namespace phmm {

// The paths with per-position w and x hold 8R + ~55 registers a lane, so above R = 10
// two warps per scheduler fit; below, three.
template <int R, int W>
constexpr int tile64_min_ctas() {
    return W > 1 ? (R <= 8 ? 16 : 8) / W : (R <= 10 ? 6 : 4);
}

template <int G, int R, int W, bool GCP, bool EXT>
__global__ void __launch_bounds__(W == 1 ? kBlockThreads : 32 * W, tile64_min_ctas<R, W>())
fp64_tile_kernel(DevView v, const Task* __restrict__ items, const unsigned long long* count,
                 unsigned long long* counter, ExtList ext) {
    using T = TileWavefront<double, G, R, W, GCP, EXT>;
    extern __shared__ double2 smem64_all[];
    float* ph = reinterpret_cast<float*>(smem64_all);  // 128 probabilities
    double2* smem64 = smem64_all + 32;
    for (int i = threadIdx.x; i < 128; i += blockDim.x) ph[i] = v.ph2pr[i];
    __syncthreads();
    constexpr int kWarps = T::kWarps;
    static_assert(T::kBlockGroup || kWarps == kWarpsPerBlock, "independent warps");
    const int warp = threadIdx.x >> 5;
    const int lane = threadIdx.x & 31;
    auto* tab = reinterpret_cast<typename T::Word*>(smem64) + warp * T::kTableWords;
    auto* ring = reinterpret_cast<typename T::RingRow*>(reinterpret_cast<char*>(smem64) + kWarps * T::kSmemBytes);
    __shared__ unsigned next;
    const unsigned n = (unsigned)*count;
    const unsigned ntasks = (n + T::NG - 1) / T::NG;
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
        x = __reduce_max_sync(kFullMask, x);  // see fp32_tile_kernel
        if (x >= ntasks) break;
        const unsigned first = x * T::NG;
        const int ntask = (int)min((unsigned)T::NG, n - first);
        const int grp = lane / G;
        const int t = lane - grp * G;
        const bool active = grp < ntask;
        const Task* item = items + first + (active ? grp : 0);
        typename T::Sum sum;
        sum.s[0] = 0.0;
        {
            const Task it = *item;
            const int H = v.hap_len[it.hap];
            const PackedHap hap(reinterpret_cast<const uint32_t*>(v.hap_code + v.hap_start[it.hap]), H);
            typename T::Reads rd;
            rd.L[0] = v.read_len[it.read];
            rd.read[0].p = v.read_pack + v.read_start[it.read];
            rd.ph = ph;
            const float eps = GCP ? ph[v.read_gcp[it.read]] : kEps;
            rd.eps[0] = (double)eps;
            rd.beta[0] = GCP ? (double)(float)(1.0 - (double)eps) : (double)kBeta;  // gpuworker.cuh:1049
            const unsigned key = v.read_meta[it.read].key;
            const unsigned kmax = __reduce_max_sync(kFullMask, key);
            const bool uni = __reduce_min_sync(kFullMask, key) == kmax && kmax != kNoKey;
            const int K = T::kBlockGroup ? 0 : (int)((__reduce_max_sync(kFullMask, (unsigned)(H + G)) + 3u) & ~3u);
            T::run(rd, hap, H, K, uni, tab, ring, nullptr, 0, t, T::kBlockGroup ? warp : 0, lane, 0.0, sum);
        }
        if (active && t == G - 1 && (!T::kBlockGroup || warp == W - 1)) {
            const volatile Task* vi = item;   // read again rather than kept over the steps
            const int read = vi->read, hap = vi->hap;
            const int64_t out = vi->out;
            const int L = v.read_len[read], H = v.hap_len[hap];
            const int e = EXT ? sum.e : kScaledExp;
            double res = -INFINITY;
            if (sum.s[0] > 0.0)
                res = log10(sum.s[0] / (double)H) - (double)e * 0.30102999566398119521 - log10((double)kTileD0);
            // gcp quality 0: beta = 0, nothing to rescale by
            const bool none = GCP && !((float)(1.0 - (double)ph[v.read_gcp[read]]) > 0.0f);
            v.scores[out] = none ? NAN : (float)res;
            if (!EXT && !none &&
                !(sum.s[0] >= scaled_tile_threshold(L, H, v.read_meta[read].range) && sum.s[0] <= DBL_MAX))
                ext.append(Task{read, hap, out});
        }
        __syncwarp();
    }
}

template <int G, int R, int W, bool GCP, bool EXT>
cudaError_t launch_fp64_tile(const Fp64LaunchArgs& a) {
    using T = TileWavefront<double, G, R, W, GCP, EXT>;
    fp64_tile_kernel<G, R, W, GCP, EXT><<<a.grid, 32 * T::kWarps, T::kBlockSmem, a.stream>>>(
        a.view, a.items, a.count, a.counter, a.ext_list);
    return cudaGetLastError();
}

template <int G, int R, int W, bool GCP, bool EXT>
Fp64Config make_tile64_config() {
    using T = TileWavefront<double, G, R, W, GCP, EXT>;
    Fp64Config c{};
    c.G = T::kLanes;
    c.R = R;
    c.ext = EXT;
    c.gcp = GCP;
    c.exact = true;
    c.per_task = T::NG;
    c.block_threads = 32 * T::kWarps;
    c.tasks_per_block = T::kBlockGroup ? 1 : T::kWarps;
    c.smem_bytes = T::kBlockSmem;
    c.kernel = reinterpret_cast<const void*>(&fp64_tile_kernel<G, R, W, GCP, EXT>);
    c.launch = &launch_fp64_tile<G, R, W, GCP, EXT>;
    return c;
}

// scaled-tier tiles G x R for R in [R0, R1], both modes
template <int G, int R0, int R1>
void register_tiles64(std::vector<Fp64Config>& out) {
    if constexpr (R0 <= R1) {
        out.push_back(make_tile64_config<G, R0, 1, false, false>());
        out.push_back(make_tile64_config<G, R0, 1, true, false>());
        register_tiles64<G, R0 + 1, R1>(out);
    }
}

// tiles over blocks of W warps: the scaled tier's, and where EXT the extended tier's too
template <int W, int R0, int R1, bool GCP, bool EXT>
void register_long64(std::vector<Fp64Config>& out) {
    if constexpr (R0 <= R1) {
        out.push_back(make_tile64_config<32, R0, W, GCP, false>());
        if constexpr (EXT) out.push_back(make_tile64_config<32, R0, W, GCP, true>());
        register_long64<W, R0 + 1, R1, GCP, EXT>(out);
    }
}

}  // namespace phmm
