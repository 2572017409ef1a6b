// Batch preparation kernels: pack reads and haplotypes into the HBM layout
// of device_common.cuh, then build the sorted work list.
//
// Work list: every item (a unit of one or two reads of a record, placed in a
// length bucket by the host, against one haplotype) gets a bin
// (bucket rank, cap - min(H, cap)), cap the batch's longest haplotype or 4095, so
// that an exclusive scan over each rank's bins followed by an atomic scatter
// sorts the items by tile bucket (largest tiles first) and, inside a bucket, by
// haplotype length descending.  Warps of the persistent kernel then take
// consecutive items, so the groups of a warp have nearly equal haplotype lengths
// (little idle work) and the longest pairs start first (short tail).  The order of pairs with the
// same bin is not deterministic; each pair still writes its own output slot,
// so results are.
#pragma once

#include "device_common.cuh"
#include "wavefront_tile.cuh"

namespace phmm {

constexpr int kHBins = 4096;     // most haplotype-length classes per bucket
constexpr int kMaxBuckets = 96;

struct PrepArgs {
    // caller arrays (device)
    const uint8_t* read_bases;
    const uint8_t* base_quals;
    const uint8_t* ins_quals;
    const uint8_t* del_quals;
    const int64_t* read_offsets;
    const int32_t* read_lengths;
    const uint8_t* hap_bases;
    const int64_t* hap_offsets;
    const int32_t* hap_lengths;
    const uint8_t* gcp_quals;       // gcp mode only (else null)
    // index arrays (device, computed on the host)
    const int32_t* read_record;     // [num_reads]
    const int32_t* read_local;      // [num_reads] read index inside its record
    const int32_t* rec_haps;        // [num_records] H
    const int64_t* rec_hap_base;    // [num_records]
    const int64_t* rec_pair_base;   // [num_records]
    const int64_t* read_start;      // [num_reads] packed start (positions)
    const int64_t* hap_start;       // [num_haps] packed start (bytes)
    int64_t num_reads;
    int64_t num_haps;
    // outputs
    uint32_t* read_pack;
    uint8_t* hap_code;
    uint8_t* read_gcp;              // [num_reads], gcp mode only (else null)
    ReadMeta* read_meta;            // what the exact-tile kernels need per read
    const float* ph2pr;             // 128 probabilities
};

// Byte fills of up to kFillRanges device ranges (4-byte aligned, whole words) by
// the pack kernel's first blocks.  Not memset nodes: a copy engine may run those,
// where they queue behind other streams' pending copies.
constexpr int kFillRanges = 4;
struct FillArgs {
    uint32_t* ptr[kFillRanges];
    long long words[kFillRanges];
    uint32_t value[kFillRanges];
};

#ifdef PHMM_PREP_KERNELS_IMPL
__device__ __forceinline__ uint32_t pack_position(uint32_t base, uint32_t bq, uint32_t iq, uint32_t dq) {
    bq = bq > 127u ? 127u : bq;
    iq = iq > 127u ? 127u : iq;
    dq = dq > 127u ? 127u : dq;
    return code_of((uint8_t)base) | (bq << 8) | (iq << 16) | (dq << 24);
}

// One launch prepares a batch's arrays: the first fill_blocks blocks fill, the
// next read_blocks pack reads, the rest pack haplotypes.  As three launches the
// stage's chain was two launch gaps longer, which is most of the time of a call
// of one small region (see hist_scan_kernel for the stage's figures).
// Warp per read; a lane packs 4 consecutive positions and stores them as one
// 16-byte word group.  Where the four source arrays are 4-byte aligned at the
// read's offset, whole groups inside the read are read with one 4-byte load
// per array; the read's ragged end (and unaligned sources) go byte by byte.
// Also notes per read what the exact-tile kernels ask of all its positions.  Forming
// their coefficients here too, 16 bytes a position, was measured: 2.3 times the
// stage's time (0.11 -> 0.25 ms for 2,000 uneven regions) for 1% of the FP32 stage's.
__device__ __forceinline__ void pack_reads(const PrepArgs& a, const float* ph, int64_t block, int64_t nblocks) {
    const int64_t warp = (block * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (nblocks * blockDim.x) >> 5;
    const int lane = threadIdx.x & 31;
    for (int64_t i = warp; i < a.num_reads; i += nwarps) {
        const int L = a.read_lengths[i];
        const int Lp = (L + 3) & ~3;
        const int64_t src = a.read_offsets[i];
        const uint8_t* rb = a.read_bases + src;
        const uint8_t* bq = a.base_quals + src;
        const uint8_t* iq = a.ins_quals + src;
        const uint8_t* dq = a.del_quals + src;
        const bool aligned = ((reinterpret_cast<uintptr_t>(rb) | reinterpret_cast<uintptr_t>(bq) |
                               reinterpret_cast<uintptr_t>(iq) | reinterpret_cast<uintptr_t>(dq)) & 3u) == 0;
        uint4* dst = reinterpret_cast<uint4*>(a.read_pack + a.read_start[i]);  // 16-byte aligned
        if (a.read_gcp && lane == 0) {
            const uint32_t g = L > 0 ? a.gcp_quals[src] : 10u;
            a.read_gcp[i] = (uint8_t)(g > 127u ? 127u : g);
        }
        float range = 0.0f, bias = 0.0f, beta = kBeta;
        uint32_t key = kNoKey, flags = 0;
        bool same = true;   // gap qualities of the lane's positions equal the first position's
        if (L > 0) {
            key = min((uint32_t)iq[0], 127u);
            if (a.gcp_quals) {
                const uint32_t g = min((uint32_t)a.gcp_quals[src], 127u);
                key |= g << 8;
                beta = (float)(1.0 - (double)ph[g]);  // gpuworker.cuh:1049
                if (!(beta >= kMinAlpha)) flags = 1u;      // gcp quality 0: nothing to rescale by
            }
        }
        const float inv_beta = 1.0f / beta;
        for (int c = lane * 4; c < Lp; c += 128) {
            uint32_t w[4];
            if (aligned && c + 3 < L) {
                const uint32_t r4 = *reinterpret_cast<const uint32_t*>(rb + c);
                const uint32_t b4 = *reinterpret_cast<const uint32_t*>(bq + c);
                const uint32_t i4 = *reinterpret_cast<const uint32_t*>(iq + c);
                const uint32_t d4 = *reinterpret_cast<const uint32_t*>(dq + c);
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    w[j] = pack_position((r4 >> (8 * j)) & 0xffu, (b4 >> (8 * j)) & 0xffu, (i4 >> (8 * j)) & 0xffu,
                                         (d4 >> (8 * j)) & 0xffu);
            } else {
#pragma unroll
                for (int j = 0; j < 4; ++j)
                    w[j] = c + j < L ? pack_position(rb[c + j], bq[c + j], iq[c + j], dq[c + j]) : 4u;
            }
            dst[c >> 2] = make_uint4(w[0], w[1], w[2], w[3]);
            {
                float d = ph[(w[0] >> 16) & 0x7fu], sg = ph[(w[0] >> 24) & 0x7fu];
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    if (c + j >= L) break;
                    same = same && (w[j] >> 16) == (key & 0xffu) * 0x101u;
                    float dn = d, sn = sg;   // past the end the last position's
                    if (c + j + 1 < L) {
                        const uint32_t in = j < 3 ? (w[j < 3 ? j + 1 : 3] >> 16) & 0x7fu : min((uint32_t)iq[c + 4], 127u);
                        const uint32_t sd = j < 3 ? (w[j < 3 ? j + 1 : 3] >> 24) & 0x7fu : min((uint32_t)dq[c + 4], 127u);
                        dn = ph[in];
                        sn = ph[sd];
                    }
                    const TileLink k = tile_link(c + j + 1 < L ? 1.0f - (dn + sn) : beta, dn, beta, inv_beta);
                    range = fmaxf(range, tile_range(k, sg));
                    bias += tile_emission_error(1.0f - ph[(w[j] >> 8) & 0x7fu], k);
                    if (!(fabsf(1.0f - (d + sg)) >= kMinAlpha)) flags |= 1u;
                    d = dn;
                    sg = sn;
                }
            }
        }
        {
            same = __all_sync(kFullMask, same);
            flags = __any_sync(kFullMask, flags != 0u) ? 1u : 0u;
            // positive floats order as their bits; an infinite or NaN bound stays the largest
            range = __uint_as_float(__reduce_max_sync(kFullMask, __float_as_uint(range)));
#pragma unroll
            for (int d = 16; d >= 1; d >>= 1) bias += __shfl_xor_sync(kFullMask, bias, d);
            if (lane == 0) {
                a.read_meta[i].bias = bias * 0.43429448f;
                a.read_meta[i].range = range;
                a.read_meta[i].key = same ? key : kNoKey;
                a.read_meta[i].flags = flags;
            }
        }
    }
}

// Warp per haplotype; a lane encodes 16 consecutive positions (4-byte loads
// where the source is 4-byte aligned and the 16 positions are inside the
// haplotype) and stores them as one 16-byte word; the padding to 16 bytes is
// code 4.
__device__ __forceinline__ void pack_haps(const PrepArgs& a, int64_t block, int64_t nblocks) {
    const int64_t warp = (block * blockDim.x + threadIdx.x) >> 5;
    const int64_t nwarps = (nblocks * blockDim.x) >> 5;
    const int lane = threadIdx.x & 31;
    for (int64_t i = warp; i < a.num_haps; i += nwarps) {
        const int H = a.hap_lengths[i];
        const int Hp = (H + 15) & ~15;
        const uint8_t* hb = a.hap_bases + a.hap_offsets[i];
        const bool aligned = (reinterpret_cast<uintptr_t>(hb) & 3u) == 0;
        uint4* dst = reinterpret_cast<uint4*>(a.hap_code + a.hap_start[i]);  // 16-byte aligned
        for (int c = lane * 16; c < Hp; c += 512) {
            uint32_t w[4];
            if (aligned && c + 15 < H) {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    const uint32_t v = *reinterpret_cast<const uint32_t*>(hb + c + 4 * q);
                    w[q] = code_of(v & 0xffu) | (code_of((v >> 8) & 0xffu) << 8) | (code_of((v >> 16) & 0xffu) << 16) |
                           (code_of(v >> 24) << 24);
                }
            } else {
#pragma unroll
                for (int q = 0; q < 4; ++q) {
                    uint32_t v = 0;
#pragma unroll
                    for (int j = 0; j < 4; ++j) {
                        const int cc = c + 4 * q + j;
                        v |= (cc < H ? code_of(hb[cc]) : 4u) << (8 * j);
                    }
                    w[q] = v;
                }
            }
            dst[c >> 4] = make_uint4(w[0], w[1], w[2], w[3]);
        }
    }
}

__global__ void __launch_bounds__(256)
pack_kernel(PrepArgs a, FillArgs f, int fill_blocks, int read_blocks) {
    __shared__ float ph[128];
    const int b = blockIdx.x;
    if (b < fill_blocks) {
        for (int k = 0; k < kFillRanges; ++k)
            for (long long i = (long long)b * blockDim.x + threadIdx.x; i < f.words[k];
                 i += (long long)fill_blocks * blockDim.x)
                f.ptr[k][i] = f.value[k];
    } else if (b < fill_blocks + read_blocks) {
        if (threadIdx.x < 128) ph[threadIdx.x] = a.ph2pr[threadIdx.x];
        __syncthreads();
        pack_reads(a, ph, b - fill_blocks, read_blocks);
    } else {
        pack_haps(a, b - fill_blocks - read_blocks, gridDim.x - fill_blocks - read_blocks);
    }
}

#endif  // PHMM_PREP_KERNELS_IMPL

// First work item of every bucket rank (and the end of the last), known to the host.
struct RankItems {
    long long begin[kMaxBuckets + 1];
};

struct BinArgs {
    const int32_t* hap_lengths;
    const int32_t* read_record;
    const int32_t* read_local;
    const int32_t* rec_haps;
    const int64_t* rec_hap_base;
    const int64_t* rec_pair_base;
    const int32_t* unit_read0;      // [num_units]
    const int32_t* unit_read1;      // [num_units], -1 for a one-read unit
    const int32_t* unit_bucket;     // [num_units]
    int64_t num_units;
    int nbuckets;
    int hcap;                       // longest haplotype class (0: all in one class, the plain form)
    int hbins;                      // haplotype-length classes per bucket: hcap + 1, up to a multiple of 4
    bool reversed;                  // bucket b's rank is nbuckets - 1 - b (largest tiles first), else b
    unsigned int* hist;             // [nbuckets * hbins]
    unsigned long long* cursor;     // [nbuckets * hbins] scatter positions
    RankItems ranks;
    Item* items;
};

__device__ __forceinline__ int bin_of(const BinArgs& a, int bucket, int H) {
    return (a.reversed ? a.nbuckets - 1 - bucket : bucket) * a.hbins + a.hcap - (H < a.hcap ? H : a.hcap);
}

#ifdef PHMM_PREP_KERNELS_IMPL
// warp-aggregated increment: lanes that hit the same counter share one atomic
template <class T>
__device__ __forceinline__ T aggregated_add(T* counter, unsigned key) {
    const unsigned active = __activemask();
    const unsigned peers = __match_any_sync(active, key);
    const int leader = __ffs(peers) - 1;
    const int lane = threadIdx.x & 31;
    T base = 0;
    if (lane == leader) base = atomicAdd(counter, (T)__popc(peers));
    base = __shfl_sync(peers, base, leader);
    return base + (T)__popc(peers & ((1u << lane) - 1u));
}

// thread per unit: histogram of (bucket, H class)
__global__ void bin_count_kernel(BinArgs a) {
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < a.num_units;
         u += (int64_t)gridDim.x * blockDim.x) {
        const int g = a.read_record[a.unit_read0[u]];
        const int nh = a.rec_haps[g];
        const int64_t hb = a.rec_hap_base[g];
        const int b = a.unit_bucket[u];
        for (int h = 0; h < nh; ++h) {
            const int bin = bin_of(a, b, a.hap_lengths[hb + h]);
            aggregated_add(&a.hist[bin], (unsigned)bin);
        }
    }
}

// thread per unit: scatter items into their sorted slots
__global__ void bin_scatter_kernel(BinArgs a) {
    for (int64_t u = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; u < a.num_units;
         u += (int64_t)gridDim.x * blockDim.x) {
        const int r0 = a.unit_read0[u], r1 = a.unit_read1[u];
        const int g = a.read_record[r0];
        const int nh = a.rec_haps[g];
        const int64_t hb = a.rec_hap_base[g];
        const int b = a.unit_bucket[u];
        const int64_t ob0 = a.rec_pair_base[g] + (int64_t)a.read_local[r0] * nh;
        const int64_t ob1 = r1 >= 0 ? a.rec_pair_base[g] + (int64_t)a.read_local[r1] * nh : -1;
        for (int h = 0; h < nh; ++h) {
            const int bin = bin_of(a, b, a.hap_lengths[hb + h]);
            const unsigned long long pos = aggregated_add(&a.cursor[bin], (unsigned)bin);
            a.items[pos] = Item{r0, r1, (int32_t)(hb + h), 0, ob0 + h, r1 >= 0 ? ob1 + h : -1};
        }
    }
}

// Exclusive scan of the histogram into cursor: block r scans the hbins bins of
// rank r from the rank's first item, which the host knows (it counts every
// bucket's items).  kHistScanThreads threads take 4 bins each per round, so loads
// and stores are whole 16- and 32-byte words; the block is small enough to find
// room on an SM next to the long-running blocks of another engine's kernels.
// One block over all ranks' 4,096 bins, 432 bins a thread, was most of the stage:
// 0.21 ms a call whatever the batch, now 0.03 ms (one region of 32 x 4 pairs).
constexpr int kHistScanThreads = 256;
__global__ void __launch_bounds__(kHistScanThreads)
hist_scan_kernel(const unsigned int* hist, unsigned long long* cursor, int hbins, RankItems items) {
    __shared__ unsigned int wsum[kHistScanThreads / 32];
    const int rank = blockIdx.x, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    if (items.begin[rank] == items.begin[rank + 1]) return;
    const unsigned int* h = hist + (long long)rank * hbins;
    unsigned long long* cur = cursor + (long long)rank * hbins;
    unsigned long long base = (unsigned long long)items.begin[rank];
    for (int b0 = 0; b0 < hbins; b0 += 4 * kHistScanThreads) {  // hbins is a multiple of 4
        const int b = b0 + 4 * tid;
        uint4 n = make_uint4(0u, 0u, 0u, 0u);
        if (b < hbins) n = *reinterpret_cast<const uint4*>(h + b);
        const unsigned int mine = n.x + n.y + n.z + n.w;
        unsigned int incl = mine;
#pragma unroll
        for (int d = 1; d < 32; d <<= 1) {
            const unsigned int y = __shfl_up_sync(kFullMask, incl, d);
            if (lane >= d) incl += y;
        }
        __syncthreads();  // the previous round's sums are read
        if (lane == 31) wsum[warp] = incl;
        __syncthreads();
        unsigned int before = 0, all = 0;
#pragma unroll
        for (int w = 0; w < kHistScanThreads / 32; ++w) {
            if (w < warp) before += wsum[w];
            all += wsum[w];
        }
        if (b < hbins) {
            const unsigned long long c0 = base + before + incl - mine;
            ulonglong2* out = reinterpret_cast<ulonglong2*>(cur + b);
            out[0] = make_ulonglong2(c0, c0 + n.x);
            out[1] = make_ulonglong2(c0 + n.x + n.y, c0 + n.x + n.y + n.z);
        }
        base += all;
    }
}

#endif  // PHMM_PREP_KERNELS_IMPL

// ---------------------------------------------------------------- FP64 list order
// The FP32 pass appends flagged pairs to the FP64 class lists in completion
// order, so the pairs of one FP64 warp task (NG of them) would have unrelated
// haplotype lengths and the warp would run as long as the longest.  A counting
// sort by haplotype length (descending, 16-position classes; longer than
// 8,175 in the last class) makes consecutive pairs alike, as the FP32 work
// list is: count, per-class scan, scatter into a second list with the same
// class offsets.
constexpr int kRescueHBins = 512;
struct RescueSortArgs {
    const Task* in;                   // class lists in append order
    Task* out;                        // the same lists, sorted
    int classes;
    const long long* off;             // [classes] list starts
    const unsigned long long* count;  // [classes] list lengths
    const int32_t* hap_len;
    unsigned int* hist;               // [classes * kRescueHBins], zeroed before the batch
    unsigned long long* cursor;       // [classes * kRescueHBins]
};

__device__ __forceinline__ int rescue_hbin(int H) {
    const int b = H >> 4;
    return kRescueHBins - 1 - (b < kRescueHBins - 1 ? b : kRescueHBins - 1);
}

#ifdef PHMM_PREP_KERNELS_IMPL
__global__ void rescue_count_kernel(RescueSortArgs a) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (int c = 0; c < a.classes; ++c) {
        const long long n = (long long)a.count[c];
        const Task* in = a.in + a.off[c];
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
            const int bin = c * kRescueHBins + rescue_hbin(a.hap_len[in[i].hap]);
            aggregated_add(&a.hist[bin], (unsigned)bin);
        }
    }
}

// one warp per class: exclusive scan of its bins (16 per lane) from the list start
__global__ void __launch_bounds__(32) rescue_scan_kernel(RescueSortArgs a) {
    constexpr int kPer = kRescueHBins / 32;
    const int c = blockIdx.x, lane = threadIdx.x;
    const unsigned int* h = a.hist + c * kRescueHBins + lane * kPer;
    unsigned long long sum = 0;
#pragma unroll
    for (int i = 0; i < kPer; ++i) sum += h[i];
    unsigned long long incl = sum;
#pragma unroll
    for (int d = 1; d < 32; d <<= 1) {
        const unsigned long long y = __shfl_up_sync(kFullMask, incl, d);
        if (lane >= d) incl += y;
    }
    unsigned long long run = (unsigned long long)a.off[c] + incl - sum;
    unsigned long long* cur = a.cursor + c * kRescueHBins + lane * kPer;
#pragma unroll
    for (int i = 0; i < kPer; ++i) {
        cur[i] = run;
        run += h[i];
    }
}

__global__ void rescue_scatter_kernel(RescueSortArgs a) {
    const long long stride = (long long)gridDim.x * blockDim.x;
    for (int c = 0; c < a.classes; ++c) {
        const long long n = (long long)a.count[c];
        const Task* in = a.in + a.off[c];
        for (long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += stride) {
            const Task t = in[i];
            const int bin = c * kRescueHBins + rescue_hbin(a.hap_len[t.hap]);
            a.out[aggregated_add(&a.cursor[bin], (unsigned)bin)] = t;
        }
    }
}
#endif  // PHMM_PREP_KERNELS_IMPL

}  // namespace phmm
