// Allocation-free forward: pairhmm_forward_pairs_noalloc.
//
// Some callers cannot allocate device memory at all: code running inside a
// host that owns every device allocation itself (a pre-sized arena, a
// framework allocator it must not bypass), or code called from a context where
// cudaMalloc/cudaFree are forbidden because they synchronise the device.  This
// entry point serves them.  The caller passes device buffers it already owns
// (read and haplotype bytes, a flat list of pairs, the score array) and the
// call allocates nothing: no cudaMalloc, no cudaFree, no allocating library
// routine, no host heap either.
//
// The kernel reads the caller's bytes directly instead of a packed copy.  A warp
// takes a few consecutive pairs of the list at a time and runs those of one shape
// together on the exact tiles of wavefront_tile.cuh: 8 lanes a pair up to 160
// positions, 16 up to 320, then 32 lanes with the read's parts in turn.  Few pairs
// take a general form in a second launch, the whole warp, 4 to 16 positions a lane by
// the read's length, longer reads in tiles of 512: reads of at most 8 positions, and,
// once more, pairs whose sum on the tiles is too small for their range (there is no
// FP64 pass behind this entry point, and the general form's range reaches further
// down).  24,600 pairs of 70-250 x 120-650 positions take 1.09 ms, against 4.0 ms with
// the general form for all (one pair on 512 positions a warp, eleven operations a
// cell); what bounds it is the instruction cache (several shapes in flight) and the
// last pairs of a short list.
// The only scratch, the per-warp border between a read's parts, lives in
// kScratchBytes of statically allocated device memory defined below: every GPU
// that loads this library holds that much memory until the process exits (the work
// queues take 8 KB more).  Limits: haplotype length up to kMaxHapLength; any read
// length.  Results are FP32 only, with no FP64 recompute of pairs whose FP32 result
// underflows (those return what FP32 gives, possibly -inf, as the reference does).
//
// Every call shares the one scratch array and it keeps the last call's
// contents.  Nothing in it has to start at zero: within a pair each border row
// is written by one tile before the next tile reads it.  Calls whose work
// overlaps on the GPU (two streams, or two host threads) race on the scratch
// and must be serialised by the caller; an overlap can spoil the scores of the
// calls that overlap (reads of several parts or tiles), never a later call's.
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <cfloat>
#include <cstdint>
#include <mutex>

#include "../../include/pairhmm_b200.h"
#include "device_common.cuh"
#include "wavefront_tile.cuh"

namespace phmm {
namespace noalloc {

constexpr int kMaxHapLength = 16384;
constexpr size_t kScratchBytes = size_t(64) << 20;  // 64 MiB
constexpr int kThreads = 64;                        // 2 warps per block
constexpr int kMaxDevices = 64;

// Border scratch: per resident warp, 2 buffers x rows x float4.
static __device__ __align__(256) float4 g_scratch[kScratchBytes / sizeof(float4)];

// probability table p(q) = float(10^(-q/10)) (gpuworker.cuh:473-486), in
// constant memory of this module, initialised in the module image itself: no
// upload, so a context that is torn down and created again has it too
static __constant__ float c_ph2pr[128] = {
#include "ph2pr_table.inc"
};

__device__ __forceinline__ uint32_t encode(uint8_t c) {
    return c == 'A' ? 0u : c == 'C' ? 1u : c == 'G' ? 2u : c == 'T' ? 3u : 4u;
}

__device__ __forceinline__ float ph_of(const float* ph, uint8_t q) { return ph[q > 127 ? 127 : q]; }

// The work queues: list positions handed out so far.  A call takes the next words in turn
// and clears them in a launch of its own ahead of its kernel, so it relies on nothing that
// an earlier call left, and calls that overlap hand out their own pairs each (a captured
// call keeps its words: its replays clear them too).
constexpr unsigned kQueues = 1024;
static __device__ unsigned g_queue[kQueues][2];   // the tiles' and the general form's

__global__ void clear_queue_kernel(unsigned queue) { g_queue[queue][0] = g_queue[queue][1] = 0; }

// Marks a pair's score between the call's two kernels: a NaN that no score is.
constexpr uint32_t kToGeneral = 0x7fa50a51u;

struct Args {
    const uint8_t *read_bases, *base_quals, *ins_quals, *del_quals, *hap_bases;
    const pairhmm_pair_t* pairs;
    int64_t num_pairs;
    float* scores;
    float4* scratch;    // per warp 2 * rows
    int64_t rows;
    int64_t nwarps;
    int max_h;
    int grab;           // pairs a warp takes at a time, at most 32
    int look;           // pairs a warp of the general form looks through at a time, at most 32
    unsigned queue;     // the call's words of g_queue
};

// A read's positions straight from the caller's arrays, as the packed words hold them.
struct ByteRead {
    const uint8_t *b, *bq, *iq, *dq;
    __device__ __forceinline__ uint32_t word(int c) const {
        auto q = [&](const uint8_t* a) { const uint32_t v = __ldg(a + c); return v > 127u ? 127u : v; };
        return encode(__ldg(b + c)) | (q(bq) << 8) | (q(iq) << 16) | (q(dq) << 24);
    }
};
struct ByteHap {
    const uint8_t* p;
    int H;
    __device__ __forceinline__ uint32_t codes(int i) const {
        uint32_t w = 0;
#pragma unroll
        for (int j = 0; j < 4; ++j) w |= encode(__ldg(p + min_i(4 * i + j, H - 1))) << (8 * j);
        return w;
    }
};

constexpr int kMaxR = 20;
// R is a multiple of 4, so a lane holds R .. R-4 positions (the read's length over the
// lanes, rounded down, may be one below the shape's smallest).  With an R for every 8
// positions some 15 shapes were in flight and the kernel waited for instructions
// (no_instruction 4.8 of 7 cycles per issue, 2.1 ms).
constexpr int kStepR = 4;
constexpr int span_of(int R) { return R > kStepR ? kStepR + 1 : R; }
constexpr int kTableBytes = 5 * (kMaxR / 4) * 32 * 16;   // per warp
constexpr int kRingBytes = 64 * 16;
constexpr size_t kSmem = (kThreads / 32) * (size_t)(kTableBytes + kRingBytes);

// Pairs `mine` (by lane: the group's pair, or -1) of one shape.  Marked for the general
// form are pairs whose sum lies so low that the tiles' rounding in the denormal range,
// which sets in earlier than the general form's (N lies 1/delta below M), could be more
// than 2^-23 of it.  That is the pair's own sum, so its form, and with it its score,
// depends on no other pair of the list.
template <int G, int R>
__device__ __noinline__ void run_tile(const Args& a, const float* ph, char* smem, float4* wscr, int64_t mine, int parts) {
    using T = TileWavefront<float, G, R, G == 32 ? 0 : 1, false, false, G == 32, ByteRead, ByteHap, span_of(R)>;
    const int lane = threadIdx.x & 31;
    const int t = lane % G;
    // groups without a pair repeat the first group's and write nothing
    const int64_t first = __shfl_sync(kFullMask, mine, 0);
    const pairhmm_pair_t pr = a.pairs[mine >= 0 ? mine : first];
    const int L = pr.read_length, H = pr.hap_length;
    typename T::Reads rd;
    rd.ph = ph;
    rd.read[0] = ByteRead{a.read_bases + pr.read_offset, a.base_quals + pr.read_offset, a.ins_quals + pr.read_offset,
                          a.del_quals + pr.read_offset};
    rd.L[0] = L;
    rd.beta[0] = kBeta;
    rd.inv_beta[0] = 1.0f / kBeta;
    // what the engine's preparation notes per read
    const uint32_t w0 = rd.read[0].word(0);
    bool same = true;
    float bias = 0.0f, range = 0.0f;
    for (int c = t; c < L; c += G) {
        const uint32_t w = rd.read[0].word(c);
        same = same && (w >> 16) == ((w0 >> 16) & 0xffu) * 0x101u;
        const TileLink k = T::link(rd, 0, c + 1);
        range = fmaxf(range, tile_range(k, ph[(w >> 24) & 0xffu]));
        bias += tile_emission_error(1.0f - ph[(w >> 8) & 0xffu], k);
    }
#pragma unroll
    for (int d = G / 2; d >= 1; d >>= 1) {
        bias += __shfl_xor_sync(kFullMask, bias, d);
        range = fmaxf(range, __shfl_xor_sync(kFullMask, range, d));
    }
    const unsigned key = (w0 >> 16) & 0xffu;
    const bool uni = __all_sync(kFullMask, same) &&
                     __reduce_min_sync(kFullMask, key) == __reduce_max_sync(kFullMask, key);
    const int K = (int)((__reduce_max_sync(kFullMask, (unsigned)(H + G)) + 3u) & ~3u);
    typename T::Sum sum;
    sum.s[0] = 0.0;
    auto* tab = reinterpret_cast<typename T::Word*>(smem);
    static_assert(T::kSmemBytes <= kTableBytes && (G < 32 || T::kRing * sizeof(typename T::RingRow) <= kRingBytes),
                  "the block's shared memory holds every shape's table and ring");
    auto* ring = reinterpret_cast<typename T::RingRow*>(smem + kTableBytes);
    const ByteHap hap{a.hap_bases + pr.hap_offset, H};
    T::run(rd, hap, H, K, uni, tab, ring, reinterpret_cast<typename T::RingRow*>(wscr), a.rows, t, 0, lane, 0.0, sum,
           parts);
    if (mine >= 0 && t == G - 1) {
        const bool kept = sum.s[0] >= (double)tile_rounding(L, H, range) && sum.s[0] <= (double)FLT_MAX;
        a.scores[mine] = kept ? (float)(log10(sum.s[0] / (double)H) - log10((double)kTileD0) -
                                        (double)(bias * 0.43429448f))
                              : __uint_as_float(kToGeneral);
    }
    __syncwarp();
}

// The general form: one pair on the warp, R positions a lane, read tiles of 32 * R, beta
// absorbed into I and D (M keeps alpha, so no division and no degenerate-alpha case):
//   M(j,c)  = lambda*(alpha_c*M(j-1,c-1) + It(j-1,c-1) + Dt(j-1,c-1))
//   It(j,c) = eps_c*It(j,c-1) + beta*delta_c*M(j,c-1)
//   Dt(j,c) = beta*sigma_c*M(j-1,c) + eps*Dt(j-1,c)
template <int R>
__device__ __noinline__ void run_general(const Args& a, const float* ph, float4* wscr, int64_t pi) {
    constexpr int T = 32 * R;
    const int t = threadIdx.x & 31;
    const int64_t rows = a.rows;
    float* const scores = a.scores;
    {
        const pairhmm_pair_t pr = a.pairs[pi];
        const int L = pr.read_length, H = pr.hap_length;
        const uint8_t* rb = a.read_bases + pr.read_offset;
        const uint8_t* bq = a.base_quals + pr.read_offset;
        const uint8_t* iq = a.ins_quals + pr.read_offset;
        const uint8_t* dq = a.del_quals + pr.read_offset;
        const uint8_t* hb = a.hap_bases + pr.hap_offset;
        const int ntiles = (L + T - 1) / T;
        const float Dbound = kBeta * (kScale / (float)H);
        double acc = 0.0;  // summed in double: up to 16384 rows of similar size
        int rlane = -1;
        for (int tile = 0; tile < ntiles; ++tile) {
            const bool last = tile == ntiles - 1;
            const int p0 = tile * T + t * R;
            float lm[R], lx[R], alpha[R], dlt[R], sig[R], eps[R], M[R], D[R];
            uint32_t xc[R];
#pragma unroll
            for (int r = 0; r < R; ++r) {
                const int c = p0 + r;
                const bool in = c < L;
                const float p = in ? ph_of(ph, bq[c]) : 1.0f;
                const float d = in ? ph_of(ph, iq[c]) : 0.0f;
                const float sg = in ? ph_of(ph, dq[c]) : 0.0f;
                xc[r] = in ? encode(rb[c]) : 4u;
                lm[r] = in ? 1.0f - p : 0.0f;
                lx[r] = in ? p / 3.0f : 0.0f;
                alpha[r] = 1.0f - (d + sg);
                dlt[r] = in ? kBeta * d : (c == L ? kBeta : 0.0f);
                sig[r] = kBeta * sg;
                eps[r] = in ? kEps : 1.0f;
                M[r] = 0.f;
                D[r] = 0.f;
            }
            int t_res = 0, r_res = 0;
            if (last) {
                const int rel = L - 1 - tile * T;
                t_res = rel / R;
                r_res = rel - t_res * R;
            }
            const int kg = last ? H + t_res : H + 32 - 1;
            const bool res_lane = last && t == t_res;
            const bool addM = r_res == R - 1;
            if (res_lane) rlane = t;
            float4* ein = wscr + ((tile - 1) & 1) * rows;
            float4* eout = wscr + (tile & 1) * rows;
            const bool writer = !last && t == 32 - 1;
            float Ml = 0.f, Dl = 0.f, Mul = 0.f, Dul = 0.f, Iul = 0.f;
            if (t == 0 && tile == 0) { Dl = Dbound; Dul = Dbound; }
            uint32_t h = 4u;
            uint8_t base = t == 0 ? hb[0] : 0;   // of the next step, a step ahead of its use
            for (int k = 0; k <= kg; ++k) {
                uint32_t hn = __shfl_up_sync(kFullMask, h, 1);
                if (t == 0) hn = k < H ? encode(base) : 4u;
                h = hn;
                if (t == 0 && k + 1 < H) base = __ldg(hb + k + 1);
                float Mdiag = Mul, Idiag = Iul, Xdiag = Iul + Dul;
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const float lam = (xc[r] == 4u || h == 4u || xc[r] == h) ? lm[r] : lx[r];
                    const float Mold = M[r];
                    const float Dold = D[r];
                    M[r] = lam * fmaf(alpha[r], Mdiag, Xdiag);
                    D[r] = fmaf(sig[r], Mold, kEps * Dold);
                    const float In = fmaf(eps[r], Idiag, dlt[r] * Mdiag);
                    Mdiag = Mold;
                    Idiag = In;
                    Xdiag = In + Dold;
                }
                float a = Idiag;
                if (addM && k < kg) a = fmaf(kBeta, M[R - 1], a);
                acc += (double)(res_lane ? a : 0.f);
                if (writer) {
                    const int j = k - (32 - 1);
                    if (j >= 0 && j < H) *reinterpret_cast<float2*>(eout + j) = make_float2(M[R - 1], D[R - 1]);
                    if (j >= 1 && j - 1 < H) reinterpret_cast<float*>(eout + (j - 1))[2] = Idiag;
                }
                Mul = Ml;
                Dul = Dl;
                Ml = __shfl_up_sync(kFullMask, M[R - 1], 1);
                Dl = __shfl_up_sync(kFullMask, D[R - 1], 1);
                Iul = __shfl_up_sync(kFullMask, Idiag, 1);
                if (t == 0) {
                    if (tile > 0) {
                        // the border is indexed by row and feeds the next diagonal directly
                        if (k < H) {
                            const float4 b = __ldcg(ein + k);
                            Mul = b.x;
                            Dul = b.y;
                            Iul = b.z;
                        } else {
                            Mul = 0.f;
                            Dul = 0.f;
                            Iul = 0.f;
                        }
                    } else {
                        Ml = 0.f;
                        Dl = Dbound;
                        Iul = 0.f;
                    }
                }
            }
            __syncwarp();
        }
        if (t == rlane) scores[pi] = (float)(log10(acc) - (log10((double)kScale) + log10((double)kBeta)));
    }
}

// Shape of a pair's tile: 0 general, else lanes << 8 | positions a lane.
__device__ __forceinline__ int shape_of(int L) {
    if (L <= 8) return 0;   // 8 lanes of at least one position
    const int G = L <= 160 ? 8 : L <= 320 ? 16 : 32;
    const int lanes = G * (G == 32 ? (L + 32 * kMaxR - 1) / (32 * kMaxR) : 1);
    return (G << 8) | (((L + lanes - 1) / lanes + kStepR - 1) / kStepR * kStepR);
}

template <int G, int R0, int R1>   // R0, R0 + kStepR, .. R1
__device__ __forceinline__ void run_shape(const Args& a, const float* ph, char* smem, float4* wscr, int64_t mine, int R,
                                          int parts) {
    if constexpr (R0 < R1) {
        if (R != R0) return run_shape<G, R0 + kStepR, R1>(a, ph, smem, wscr, mine, R, parts);
    }
    run_tile<G, R0>(a, ph, smem, wscr, mine, parts);
}

__global__ void __launch_bounds__(kThreads, 6) forward_pairs_kernel(Args a) {
    __shared__ float ph[128];
    extern __shared__ float4 smem_all[];
    for (int i = threadIdx.x; i < 128; i += blockDim.x) ph[i] = c_ph2pr[i];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    char* const smem = reinterpret_cast<char*>(smem_all) + (threadIdx.x >> 5) * (kTableBytes + kRingBytes);
    float4* const wscr = a.scratch + warp * 2 * a.rows;
    while (warp < a.nwarps) {  // the scratch holds borders for nwarps warps only
        unsigned x = 0;
        if (lane == 0) x = atomicAdd(&g_queue[a.queue][0], 1u);
        x = __reduce_max_sync(kFullMask, x);
        const int64_t p0 = (int64_t)x * a.grab;
        if (p0 >= a.num_pairs) break;
        const int64_t pi = p0 + lane;
        int L = 0, H = 0;
        bool ok = lane < a.grab && pi < a.num_pairs;
        if (ok) {
            L = a.pairs[pi].read_length;
            H = a.pairs[pi].hap_length;
            if (L < 1 || H < 1 || H > a.max_h) {  // H beyond the declared bound would overrun the border rows
                a.scores[pi] = NAN;
                ok = false;
            }
        }
        const int shape = ok ? shape_of(L) : -1;
        unsigned left = __ballot_sync(kFullMask, ok);
        while (left) {
            const int lead = __ffs(left) - 1;
            const int sh = __shfl_sync(kFullMask, shape, lead);
            const int G = sh >> 8, R = sh & 0xff;
            const unsigned alike = __ballot_sync(kFullMask, ok && shape == sh) & left;
            // group g takes the g-th of the pairs of this shape, up to as many as the warp has groups
            const int groups = G ? 32 / G : 1;
            const int g = G ? lane / G : 0;
            unsigned pick = alike, taken = 0;
            int64_t mine = -1;
            for (int i = 0; i < groups && pick; ++i) {
                const int l = __ffs(pick) - 1;
                pick &= pick - 1;
                taken |= 1u << l;
                if (i == g) mine = p0 + l;
            }
            left &= ~taken;
            const int parts = G == 32 ? (__shfl_sync(kFullMask, L, lead) + 32 * kMaxR - 1) / (32 * kMaxR) : 1;
            if (G == 8) run_shape<8, 4, 20>(a, ph, smem, wscr, mine, R, 1);
            else if (G == 16) run_shape<16, 12, 20>(a, ph, smem, wscr, mine, R, 1);
            else if (G == 32) run_shape<32, 12, 20>(a, ph, smem, wscr, mine, R, parts);
            else if (lane == 0) a.scores[mine] = __uint_as_float(kToGeneral);
            __syncwarp();
        }
    }
}

// The pairs the tiles left: a warp looks through up to 32 of the list at a time.  A launch
// of its own, not the tiles' kernel: side by side the two thrashed the instruction cache,
// and a warp's low pairs ran one after the other while other warps had none.  46,336 pairs
// of 70-250 positions, 59% of them low: 4.8 -> 3.7 ms; all low 5.2 -> 4.6 (7.8 with 16
// positions a lane for every read, instead of 4-16 by its length; 5.0 without tiles, on
// the general form alone); none low 1.71 -> 1.71.  What bounds it: a step's serial chain,
// some 430 cycles for 4 positions a lane when the warp is alone (16 short pairs, 12 of them
// low: 131 us, 97 on the general form alone).
__global__ void __launch_bounds__(kThreads, 6) general_pairs_kernel(Args a) {
    __shared__ float ph[128];
    for (int i = threadIdx.x; i < 128; i += blockDim.x) ph[i] = c_ph2pr[i];
    __syncthreads();
    const int lane = threadIdx.x & 31;
    const int64_t warp = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    float4* const wscr = a.scratch + warp * 2 * a.rows;
    while (warp < a.nwarps) {
        unsigned x = 0;
        if (lane == 0) x = atomicAdd(&g_queue[a.queue][1], 1u);
        const int64_t p0 = (int64_t)__shfl_sync(kFullMask, x, 0) * a.look;
        if (p0 >= a.num_pairs) break;
        const bool mine = lane < a.look && p0 + lane < a.num_pairs &&
                          __float_as_uint(a.scores[p0 + lane]) == kToGeneral;
        for (unsigned m = __ballot_sync(kFullMask, mine); m; m &= m - 1) {
            const int64_t pi = p0 + __ffs(m) - 1;
            const int L = a.pairs[pi].read_length;   // warp-uniform
            if (L <= 128) run_general<4>(a, ph, wscr, pi);
            else if (L <= 192) run_general<6>(a, ph, wscr, pi);
            else if (L <= 256) run_general<8>(a, ph, wscr, pi);
            else if (L <= 384) run_general<12>(a, ph, wscr, pi);
            else run_general<16>(a, ph, wscr, pi);
            __syncwarp();
        }
    }
}

// per-device set-up: the scratch array's device address and the grid size
struct DeviceState {
    std::atomic<int> ready{0};
    std::atomic<float4*> scratch{nullptr};
    std::atomic<unsigned> calls{0};   // queue words given out
    int max_warps = 0;
};
DeviceState g_state[kMaxDevices];
std::mutex g_setup_mutex;

// Runs once per device, with that device current (the caller makes it so):
// looks up the scratch array's device address (in host code the array's name
// is only a host-side stand-in) and sizes the grid from the SM count and the
// kernel's occupancy.  Nothing here allocates.
pairhmm_status_t setup(int device, DeviceState& st) {
    std::lock_guard<std::mutex> lk(g_setup_mutex);
    if (st.ready.load()) return PAIRHMM_OK;
    float4* addr = nullptr;
    if (cudaGetSymbolAddress(reinterpret_cast<void**>(&addr), g_scratch) != cudaSuccess || addr == nullptr)
        return PAIRHMM_ERR_CUDA;
    st.scratch.store(addr);
    int sms = 0, per_sm = 0;
    if (cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device) != cudaSuccess) return PAIRHMM_ERR_CUDA;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, forward_pairs_kernel, kThreads, kSmem) != cudaSuccess ||
        per_sm < 1)
        per_sm = 1;
    st.max_warps = sms * per_sm * (kThreads / 32);
    st.ready.store(1);
    return PAIRHMM_OK;
}

}  // namespace noalloc
}  // namespace phmm

extern "C" pairhmm_status_t pairhmm_forward_pairs_noalloc(
    int32_t device, const uint8_t* read_bases, const uint8_t* base_quals, const uint8_t* ins_quals,
    const uint8_t* del_quals, const uint8_t* hap_bases, const pairhmm_pair_t* pairs, int64_t num_pairs,
    int32_t max_hap_length, float* scores, void* stream) {
    using namespace phmm::noalloc;
    if (num_pairs < 0 || device < 0 || device >= kMaxDevices) return PAIRHMM_ERR_INVALID_ARGUMENT;
    if (max_hap_length > kMaxHapLength) return PAIRHMM_ERR_LIMIT;  // the scratch is sized for 16384
    if (max_hap_length < 1) return PAIRHMM_ERR_INVALID_ARGUMENT;
    if (num_pairs == 0) return PAIRHMM_OK;
    if (!read_bases || !base_quals || !ins_quals || !del_quals || !hap_bases || !pairs || !scores)
        return PAIRHMM_ERR_INVALID_ARGUMENT;
    int prev = -1;
    if (cudaGetDevice(&prev) != cudaSuccess) return PAIRHMM_ERR_CUDA;
    if (prev != device && cudaSetDevice(device) != cudaSuccess) return PAIRHMM_ERR_CUDA;
    DeviceState& st = g_state[device];
    pairhmm_status_t status = st.ready.load() ? PAIRHMM_OK : setup(device, st);
    // the set-up's address is checked against a fresh lookup on every call (a
    // symbol lookup, no allocation): after the context was torn down and created
    // again the module, and the array with it, may sit elsewhere
    float4* scratch = nullptr;
    if (status == PAIRHMM_OK &&
        (cudaGetSymbolAddress(reinterpret_cast<void**>(&scratch), g_scratch) != cudaSuccess || !scratch))
        status = PAIRHMM_ERR_CUDA;
    if (status == PAIRHMM_OK && scratch != st.scratch.load()) st.scratch.store(scratch);
    if (status == PAIRHMM_OK) {
        // border rows per buffer for this call, and how many warps the scratch holds
        const int64_t rows = ((int64_t)max_hap_length + 2 * 32 + 8 + 63) / 64 * 64;
        const int64_t per_warp = 2 * rows * (int64_t)sizeof(float4);
        int64_t warps = (int64_t)(kScratchBytes / (size_t)per_warp);
        if (warps > st.max_warps) warps = st.max_warps;
        if (warps > num_pairs) warps = num_pairs;
        const int64_t warps_per_block = kThreads / 32;
        const int grid = (int)((warps + warps_per_block - 1) / warps_per_block);
        // pairs a warp takes at a time: a few, so that those of one read's haplotypes run
        // together, but at least four times per warp, so that the last ones end together
        int grab = (int)(num_pairs / (4 * warps));
        grab = grab < 1 ? 1 : grab > 8 ? 8 : grab;
        // the general form's: one pair each for a short list, since any may be low
        const int look = (int)std::min<int64_t>(32, std::max<int64_t>(1, num_pairs / (8 * warps)));
        Args ka{read_bases, base_quals, ins_quals, del_quals, hap_bases, pairs, num_pairs, scores,
                scratch,    rows,       warps,     max_hap_length, grab, look, st.calls.fetch_add(1) % kQueues};
        void *args[] = {&ka}, *queue[] = {&ka.queue};
        // cudaLaunchKernel returns this launch's own status, so an error the caller
        // left pending is neither reported as ours nor cleared
        cudaError_t le = cudaLaunchKernel(reinterpret_cast<const void*>(&clear_queue_kernel), dim3(1), dim3(1), queue,
                                          0, static_cast<cudaStream_t>(stream));
        if (le == cudaSuccess)
            le = cudaLaunchKernel(reinterpret_cast<const void*>(&forward_pairs_kernel), dim3(grid), dim3(kThreads),
                                  args, kSmem, static_cast<cudaStream_t>(stream));
        if (le == cudaSuccess)
            le = cudaLaunchKernel(reinterpret_cast<const void*>(&general_pairs_kernel), dim3(grid), dim3(kThreads),
                                  args, 0, static_cast<cudaStream_t>(stream));
        if (le != cudaSuccess) {
            cudaGetLastError();  // the failed launch's own error, recorded by the runtime as well
            status = PAIRHMM_ERR_CUDA;
        }
    }
    if (prev != device) cudaSetDevice(prev);
    return status;
}
