// Exact-tile wavefront: the PairHMM forward recurrence for reads whose length
// lies in (NL*(R-1), NL*R], NL the lanes of a group, so that every lane holds R
// or R-1 read positions and no position is padding.
//
// What bounds the cell.  A scheduler reads two 32-bit register operands per lane
// and cycle: an FFMA with three distinct register operands runs at 0.64 of the
// FMA peak, one with two (the third an immediate, a constant or a uniform
// register) at 0.95; FFMA2 and DFMA alike (measured with dependent-chain loops of
// each form).  The five-instruction cell of wavefront_fp32.cuh reads 13 operands,
// 6.5 cycles, and ran at 0.60-0.63 of the pipe, scalar or packed.  So the
// recurrence is scaled here for few register operands, not few instructions:
//   I unscaled (true I times the pair's scale), eps an immediate
//   N = n_c*M with n_c = delta_{c+1}, so that what N feeds into the next column's I
//       has weight 1 (in FP32 the n that the rounded w below stands for)
//   D^ = D/d_c with d_c = sigma_c/n_c, so that what N feeds into D has weight 1
//     P(j,c)  = w_c*N(j-1,c-1) + X(j,c-1)      w_c = alpha_c/(beta*delta_c)
//     N(j,c)  = l_c(h_j)*P(j,c)                l_c = beta*n_c*lambda
//     I^(j,c) = eps*I^(j,c-1) + N(j-1,c-1)     (I one row behind, as in the reference)
//     X(j,c)  = x_c*D^(j-1,c) + I^(j,c)        x_c = d_c
//     D^(j,c) = eps*D^(j-1,c) + N(j-1,c)
// 12 operands a cell, and 10 for reads whose gap-open qualities have one value at
// every position, for insertions and deletions alike (the usual case): w comes from
// a uniform register and x is 1.  A warp decides per task; both paths do the same
// arithmetic, so a pair's result does not depend on which one ran, nor on the
// group's shape: every cell, and the order of the result's sum, is the same for
// all G, R and W.
//
// Exact lanes.  The eps of I being a constant, I cannot be carried unchanged
// through padding behind the read's end.  Lanes t < m = L - NL*(R-1) hold R
// positions, the others R-1; a lane hands on the values of its last position (one
// select per value).  The last lane of the group always holds the read's end, so
//     T(j) = w_L*N(j,L-1) + I^(j+1,L-1) = M(j,L-1) + I(j,L-1),   w_L = 1/n_{L-1}
// is added up there and nowhere else.  4 % less of the uneven workload's cells are
// padding than with tiles of a multiple of 16 positions.
//
// Range (FP32).  N lies 1/delta below M (2^13 at gap quality 40), which costs the
// low end of the range; the boundary D enters as FLT_MAX/8 instead of
// (FLT_MAX/16)/H, which gives most of it back.  See tile_threshold.
//
// W > 1: reads beyond one warp's tile, the group's lanes being those of W warps.
//   Block groups: the W warps of a block.  Warp v runs kLag blocks of kBlock steps
//   behind warp v-1 and takes that warp's last column, row by row, from a ring in
//   shared memory; a block barrier after every kBlock steps is the only
//   synchronisation.  For batches of few pairs: a pair takes 1/W of the time.
//   SERIAL: one warp runs the W parts in turn, the last column of each going to the
//   next through global memory (L2), fetched 32 rows at a time into a shared ring.
//   For batches that fill the chip: no barriers, no pipeline to fill, and a pair that
//   will not reach the pass's threshold stops at the first part's end: every path to
//   the result leaves a column once and nothing on it exceeds 1, so the sum is at
//   most the mass sum_j (M + I + D)(j) on the column; below half the threshold the
//   sum would fail it too.
// Both do the same arithmetic as one group of 32*W lanes.
#pragma once

#include <climits>
#include <type_traits>

#include "device_common.cuh"

namespace phmm {

// Arithmetic of a lane's value: one pair in FP32 or FP64, or two pairs that share
// a haplotype in packed FP32 (x = read A, y = read B).
template <class V>
struct LaneOps;

template <>
struct LaneOps<float> {
    using S = float;
    static constexpr int kSides = 1;
    __device__ __forceinline__ static float make(float a, float) { return a; }
    __device__ __forceinline__ static float fma(float a, float b, float c) { return fmaf(a, b, c); }
    __device__ __forceinline__ static float mul(float a, float b) { return a * b; }
    __device__ __forceinline__ static float add(float a, float b) { return a + b; }
    __device__ __forceinline__ static float up(float v, int G) { return __shfl_up_sync(kFullMask, v, 1, G); }
    __device__ __forceinline__ static float sel(const bool (&p)[1], float a, float b) { return p[0] ? a : b; }
    // the value all lanes (and sides) hold, in a uniform register
    __device__ __forceinline__ static float uniform(float v) {
        return __uint_as_float(__reduce_max_sync(kFullMask, __float_as_uint(v)));
    }
    __device__ __forceinline__ static float side(float v, int) { return v; }
    __device__ __forceinline__ static void reload(const void* p, float (&v)[4]) {
        asm volatile("ld.volatile.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v[0]), "=f"(v[1]), "=f"(v[2]), "=f"(v[3])
                     : "r"((uint32_t)__cvta_generic_to_shared(p)));
    }
};

template <>
struct LaneOps<float2> {
    using S = float;
    static constexpr int kSides = 2;
    __device__ __forceinline__ static float2 make(float a, float b) { return make_float2(a, b); }
    __device__ __forceinline__ static float2 fma(float2 a, float2 b, float2 c) { return __ffma2_rn(a, b, c); }
    __device__ __forceinline__ static float2 mul(float2 a, float2 b) { return __fmul2_rn(a, b); }
    __device__ __forceinline__ static float2 add(float2 a, float2 b) { return __fadd2_rn(a, b); }
    __device__ __forceinline__ static float2 up(float2 v, int G) {
        return make_float2(__shfl_up_sync(kFullMask, v.x, 1, G), __shfl_up_sync(kFullMask, v.y, 1, G));
    }
    __device__ __forceinline__ static float2 sel(const bool (&p)[2], float2 a, float2 b) {
        return make_float2(p[0] ? a.x : b.x, p[1] ? a.y : b.y);
    }
    __device__ __forceinline__ static float2 uniform(float2 v) {
        const float u = LaneOps<float>::uniform(v.x);
        return make_float2(u, u);
    }
    __device__ __forceinline__ static float side(float2 v, int s) { return s ? v.y : v.x; }
    __device__ __forceinline__ static void reload(const void* p, float2 (&v)[2]) {
        asm volatile("ld.volatile.shared.v4.f32 {%0, %1, %2, %3}, [%4];"
                     : "=f"(v[0].x), "=f"(v[0].y), "=f"(v[1].x), "=f"(v[1].y)
                     : "r"((uint32_t)__cvta_generic_to_shared(p)));
    }
};

template <>
struct LaneOps<double> {
    using S = double;
    static constexpr int kSides = 1;
    __device__ __forceinline__ static double make(double a, double) { return a; }
    __device__ __forceinline__ static double fma(double a, double b, double c) { return ::fma(a, b, c); }
    __device__ __forceinline__ static double mul(double a, double b) { return a * b; }
    __device__ __forceinline__ static double add(double a, double b) { return a + b; }
    __device__ __forceinline__ static double up(double v, int G) { return __shfl_up_sync(kFullMask, v, 1, G); }
    __device__ __forceinline__ static double sel(const bool (&p)[1], double a, double b) { return p[0] ? a : b; }
    __device__ __forceinline__ static double uniform(double v) {
        const unsigned lo = __reduce_max_sync(kFullMask, (unsigned)__double2loint(v));
        const unsigned hi = __reduce_max_sync(kFullMask, (unsigned)__double2hiint(v));
        return __hiloint2double((int)hi, (int)lo);
    }
    __device__ __forceinline__ static double side(double v, int) { return v; }
};

// 2^k as a double for k clamped to the normal range (exact power of two)
__device__ __forceinline__ double pow2i(int k) {
    k = k < -1022 ? -1022 : (k > 1023 ? 1023 : k);
    return __longlong_as_double((long long)(k + 1023) << 52);
}

// Boundary value of D (times beta it is what the first column receives); the
// pair's scale is kTileD0 * H, D being 1/H there.
constexpr float kTileD0 = FLT_MAX / 8.0f;
// FP64, scaled tier: D enters 2^836 higher (near 2^961, which leaves 2^62 of headroom).
constexpr int kScaledExp = 836;
constexpr double kScaled = 0x1p836;

// Smallest sum of T that rounding in the denormal range leaves good to 2^-23: N, I and
// D^ each round by at most 2^-150 there; as terms of T they weigh at most 1/n, 1 and d,
// range being the read's largest 1/n + 2*(1 + d) (tile_range of its positions), and every
// path reaches the last position at most once.
__device__ __forceinline__ float tile_rounding(int L, int H, float range) {
    return (float)L * (float)H * 0x1p-127f * range;
}

// Smallest sum of T the FP32 pass keeps.  The second term is rescue_threshold in this
// scale (the sum there is beta*T, beta the read's own in gcp mode, over (FLT_MAX/16)/H): no
// pair that wavefront_fp32.cuh would pass on is kept here.
__device__ __forceinline__ float tile_threshold(int L, int H, float range, float beta) {
    const float cells = (float)L * (float)H * 0x1p-127f;
    return fmaxf(tile_rounding(L, H, range), 3.0f * cells * (float)H * (2.0f / beta));
}

// Smallest sum the FP64 pass's scaled tier keeps: the same terms each round by at most
// 2^-1075 in the subnormal range, so above this the sum is exact to about 2^-44.
__device__ __forceinline__ double scaled_tile_threshold(int L, int H, float range) {
    return (double)L * (double)H * (double)range * 0x1p-1030;
}

// FP32 coefficients of a column boundary: w of a position from its alpha and gap-open
// probability d, and g = beta*n of the position before it (with e, what g lacks of
// alpha/w in single precision).  l takes n from the rounded w of the next column, so
// that w and l multiply to alpha*lambda up to l's own rounding: where every position
// has the same gap quality a rounding of both would add up along the read.  For the
// same reason w may come from approximate reciprocals (two instead of four divisions a
// position: gcp mode with per-read gcp qualities 8.28 -> 7.7 ms of FP32 stage).  Past
// the read's end alpha is beta and d the last position's.
struct TileLink {
    float w, g, e, id;   // id = 1/d
};
__device__ __forceinline__ TileLink tile_link(float a, float d, float beta, float inv_beta) {
    const float id = __fdividef(1.0f, d);
    TileLink k{a * (id * inv_beta), beta * d, 0.0f, id};
    if (k.w != 0.0f) {
        const float rw = __fdividef(1.0f, k.w);
        k.g = a * rw;
        k.e = fmaf(-k.g, k.w, a) * rw;
    }
    return k;
}

// A position's share of a read's range: k the boundary behind it, sg its deletion
// gap-open probability.
__device__ __forceinline__ float tile_range(const TileLink& k, float sg) {
    return k.id + 2.0f * (1.0f + sg * k.id);
}

// l of a match (pm = 1 - p) or mismatch (pm = p/3), rounded once.
__device__ __forceinline__ float tile_emission(float pm, const TileLink& next) {
    return fmaf(pm, next.g, pm * next.e);
}
// Relative error of that rounding.  A read of few distinct qualities has few distinct
// errors, which add up along the path of matches (250 bases of quality 35-41: 9e-7 of
// log10 on average); their sum is taken off the score.
__device__ __forceinline__ float tile_emission_error(float pm, const TileLink& next) {
    const float l = tile_emission(pm, next);
    return l != 0.0f ? -__fdividef(fmaf(pm, next.g, -l) + pm * next.e, l) : 0.0f;
}

// What the preparation notes per read.
struct ReadMeta {
    float range;     // see tile_threshold
    uint32_t key;    // gap quality | gcp << 8 where insertions and deletions have the one quality at
                     // every position, else kNoKey
    uint32_t flags;  // bit 0: some |alpha| < kMinAlpha, the FP64 pass computes the read's pairs
    float bias;      // log10 of what rounding the match l of every position did to their product
};
static_assert(sizeof(ReadMeta) == 16, "ReadMeta is one 16-byte word");
constexpr uint32_t kNoKey = 0xffffffffu;

// Where a group's read positions and haplotype codes come from: the batch's packed
// layout.  word(c): a position as read_pack holds it; codes(i): the codes of rows
// 4i .. 4i+3, behind the haplotype's end any codes (those rows are past the result's).
struct PackedRead {
    const uint32_t* p;
    __device__ __forceinline__ uint32_t word(int c) const { return __ldg(p + c); }
};
struct PackedHap {
    const uint32_t* p;
    int last;
    __device__ __forceinline__ PackedHap(const uint32_t* codes, int H) : p(codes), last(((H + 15) & ~15) / 4 - 1) {}
    __device__ __forceinline__ uint32_t codes(int i) const { return __ldg(p + min_i(i, last)); }
};

// EXT (FP64): a lane keeps its values as true * 2^e with its own exponent e, for
// pairs whose values span more than a double's range; see wavefront_fp64.cuh, whose
// extended tier works the same way.
// SERIAL with W = 0: the number of parts is given at run time.
// SPAN: lanes hold R .. R-SPAN+1 positions, so that one kernel takes reads of
// (NL*(R-SPAN+1), NL*R] positions, at a select more per step and value for each.
template <class V, int G, int R, int W, bool GCP, bool EXT = false, bool SERIAL = false, class Read = PackedRead,
          class Hap = PackedHap, int SPAN = 2>
struct TileWavefront {
    using O = LaneOps<V>;
    using S = typename O::S;
    static constexpr bool kDouble = std::is_same<S, double>::value;
    static_assert(W == 1 || G == 32, "a group of several warps fills them");
    static constexpr bool kParts = W > 1 || SERIAL;   // a group may have several parts
    static_assert(SPAN >= 2 && R >= SPAN, "a lane holds at least one position");
    static_assert(!EXT || kDouble, "lane exponents go with doubles");
    static constexpr int NS = O::kSides;
    static constexpr int NG = 32 / G;    // groups per warp
    static constexpr int kLanes = G * W;  // lanes per group (0: given at run time)
    static constexpr bool kBlockGroup = W > 1 && !SERIAL;
    static_assert(!SERIAL || (W != 1 && NS == 1 && !kDouble), "serial parts: one FP32 read per warp");
    static constexpr int VN = 16 / (int)sizeof(V);     // values per 16-byte table word
    static constexpr int Q = (R + VN - 1) / VN;        // table words per lane and code
    static constexpr int kTableWords = 5 * Q * 32;     // per warp
    static constexpr int kBlock = 16;    // steps between block barriers (W > 1)
    // blocks a warp runs behind the one before it: row j leaves that warp's last lane
    // at step j + 31, and the step before row j takes it, so block b needs the other's
    // block b + 2 finished
    static constexpr int kLag = 3;
    static constexpr int kRing = 64;     // rows per ring; reader and writer are within 32 rows
    struct alignas(16) Word { V v[VN]; };
    struct alignas(16) RingRow {
        V n, i, x;
        int e;   // EXT: exponent of all three
    };
    // steps unrolled.  A batch of long reads has some 14 classes of few pairs, whose kernels
    // run side by side: at 4 steps (11 KB of code each) they thrashed the instruction cache,
    // 64 long-read regions' FP32 stage 14.6 ms against 7.0 at 2 steps and 7.9 at 1; the
    // flat list's kernel has its shapes side by side in one launch
    static constexpr int kUnroll = SERIAL || !std::is_same<Read, PackedRead>::value ? 2 : 4;
    // rows of the result summed in double one by one; else a step block's four rows in FP32
    // first (the flat list's general form sums row by row, and so do its tiles; the engine's
    // FP32 kernels sum by fours)
    static constexpr bool kRowSums = kDouble || !std::is_same<Read, PackedRead>::value;
    static constexpr int kMaxShift = 640;   // EXT: largest scale difference a hand-off converts
    static constexpr size_t kSmemBytes = (size_t)kTableWords * sizeof(Word);  // per warp, the table
    static constexpr int kWarps = kBlockGroup ? W : 2;   // per block
    // rings per block; a group's first part reads its (constant) boundary from one too,
    // so that no step branches on which part it runs
    static constexpr int kRings = kParts ? kWarps : 0;
    static constexpr int kBorderPad = 32;   // serial: row j sits at entry j + 32 of a buffer
    static constexpr size_t kBlockSmem = 128 * sizeof(float) + kWarps * kSmemBytes + kRings * kRing * sizeof(RingRow);

    struct Reads {
        const float* ph;            // the probabilities (shared memory)
        Read read[NS];
        int L[NS];
        S eps[NS];                  // GCP only
        S beta[NS];
        float inv_beta[NS];         // FP32
    };
    struct Sum {
        double s[NS];               // sum of T over the haplotype's rows, in the result lane
        int e;                      // EXT: its exponent
    };

    // Probabilities are the 32-bit model parameters, alpha, 1 - p and p/3 formed in FP32
    // as the reference forms them; FP64 forms the coefficients in double.
    struct Gap {
        float d, s;
    };
    __device__ __forceinline__ static Gap gap(const Reads& rd, int s, int c) {
        const uint32_t w = rd.read[s].word(c);
        return Gap{rd.ph[(w >> 16) & 0x7fu], rd.ph[(w >> 24) & 0x7fu]};
    }
    // the boundary before position c, c = L being the read's end
    __device__ __forceinline__ static TileLink link(const Reads& rd, int s, int c) {
        const Gap g = gap(rd, s, min_i(c, rd.L[s] - 1));
        return tile_link(c < rd.L[s] ? 1.0f - (g.d + g.s) : (float)rd.beta[s], g.d, (float)rd.beta[s], rd.inv_beta[s]);
    }

    // One warp's part of a group.  warp: its number in the group (0 where a warp holds
    // whole groups).  ring: the block's rings (block groups) or the warp's own (serial).
    // border: serial, the warp's column buffer of `rows` rows.
    // UNI: one gap quality at all positions of all the warp's reads
    template <bool UNI>
    __device__ __forceinline__ static void loop(const Reads& rd, const Hap& hap, int H, int K, Word* tab,
                                                RingRow* ring, RingRow* border, int64_t rows, int t, int warp,
                                                int parts, int lane, Sum& sum) {
        const int NL = G * parts;      // lanes of the group
        const int u = warp * 32 + t;   // lane of the group
        bool holds[SPAN - 1][NS];   // [j]: the lane holds at least R - j positions
        V wv[UNI ? 1 : R], xv[UNI ? 1 : R], N[R], D[R];
        {
            S w[NS][UNI ? 1 : R], x[NS][UNI ? 1 : R];
            float lg[NS][UNI || kDouble ? 1 : R], le[NS][UNI || kDouble ? 1 : R];
            TileLink mid[NS], last[NS];   // UNI: towards every position but the one past the end, and towards that
            int p0[NS];
#pragma unroll
            for (int s = 0; s < NS; ++s) {
                int m, base;   // m lanes hold base + 1 positions, the others base
                if constexpr (SPAN == 2) {
                    base = R - 1;
                    m = rd.L[s] - NL * base;
                } else {
                    base = rd.L[s] / NL;
                    m = rd.L[s] - NL * base;
                }
#pragma unroll
                for (int j = 0; j < SPAN - 1; ++j) holds[j][s] = base + (u < m ? 1 : 0) >= R - j;
                p0[s] = u * base + min_i(u, m);
                if constexpr (UNI) {
                    if constexpr (kDouble) {
                        const Gap g = gap(rd, s, 0);
                        w[s][0] = (double)(1.0f - (g.d + g.s)) * (1.0 / (rd.beta[s] * (double)g.d));
                    } else {
                        mid[s] = link(rd, s, 0);
                        last[s] = link(rd, s, rd.L[s]);
                        w[s][0] = mid[s].w;
                    }
                }
            }
            if constexpr (!UNI && kDouble) {
                Gap g = gap(rd, 0, min_i(p0[0], rd.L[0] - 1));
                double i = 1.0 / (rd.beta[0] * (double)g.d);
#pragma unroll
                for (int r = 0; r < R; ++r) {
                    const int c = p0[0] + r;
                    const Gap n = gap(rd, 0, min_i(c + 1, rd.L[0] - 1));   // past the end the last position's again
                    const double in = 1.0 / (rd.beta[0] * (double)n.d);
                    wv[r] = c < rd.L[0] ? (double)(1.0f - (g.d + g.s)) * i : 0.0;
                    xv[r] = c >= rd.L[0] ? 0.0 : g.s == n.d ? 1.0 : rd.beta[0] * (double)g.s * in;
                    g = n;
                    i = in;
                }
            }
            if constexpr (!UNI && !kDouble) {
#pragma unroll
                for (int s = 0; s < NS; ++s) {
                    Gap g = gap(rd, s, min_i(p0[s], rd.L[s] - 1));
                    w[s][0] = link(rd, s, min_i(p0[s], rd.L[s])).w;
#pragma unroll
                    for (int r = 0; r < R; ++r) {
                        const int c = p0[s] + r;
                        const TileLink k = link(rd, s, min_i(c + 1, rd.L[s]));
                        const Gap n = gap(rd, s, min_i(c + 1, rd.L[s] - 1));
                        x[s][r] = c >= rd.L[s] ? 0.0f : g.s == n.d ? 1.0f : g.s * k.id;
                        if (r + 1 < R) w[s][r + 1 < R ? r + 1 : r] = k.w;
                        lg[s][r] = k.g;
                        le[s][r] = k.e;
                        g = n;
                    }
                }
                // w and x go through the lane's table slots once: otherwise ptxas put the pairs
                // together from their halves again at every step (three moves a position, a
                // quarter of the step)
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    Word ww, xw;
#pragma unroll
                    for (int k = 0; k < VN; ++k) {
                        const int r = q * VN + k < R ? q * VN + k : R - 1;
                        ww.v[k] = O::make(w[0][r], w[NS - 1][r]);
                        xw.v[k] = O::make(x[0][r], x[NS - 1][r]);
                    }
                    tab[q * 32 + lane] = ww;
                    tab[(Q + q) * 32 + lane] = xw;
                }
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    V ww[VN], xw[VN];
                    O::reload(tab + q * 32 + lane, ww);
                    O::reload(tab + (Q + q) * 32 + lane, xw);
#pragma unroll
                    for (int k = 0; k < VN; ++k)
                        if (q * VN + k < R) {
                            wv[q * VN + k] = ww[k];
                            xv[q * VN + k] = xw[k];
                        }
                }
            }
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                Word words[5];
#pragma unroll
                for (int k = 0; k < VN; ++k) {
                    const int r = q * VN + k;
                    S l[NS][5];
#pragma unroll
                    for (int s = 0; s < NS; ++s) {
                        S lm = 0, lx = 0;
                        uint32_t code = 0;
                        const int c = p0[s] + r;
                        if (r < R && c < rd.L[s]) {
                            const uint32_t word = rd.read[s].word(c);
                            code = word & 0xffu;
                            const float p = rd.ph[(word >> 8) & 0x7fu];
                            const float pm = 1.0f - p;    // pairhmm_kernels.cuh:1244
                            const float px = p / 3.0f;    // pairhmm_kernels.cuh:1250
                            if constexpr (kDouble) {
                                const double n = rd.beta[0] * (double)gap(rd, 0, min_i(c + 1, rd.L[0] - 1)).d;
                                lm = (double)pm * n;
                                lx = (double)px * n;
                            } else {
                                const bool end = c + 1 >= rd.L[s];
                                TileLink k = end ? last[s] : mid[s];
                                if constexpr (!UNI) {
                                    k.g = lg[s][r < R ? r : 0];
                                    k.e = le[s][r < R ? r : 0];
                                }
                                lm = tile_emission(pm, k);
                                lx = tile_emission(px, k);
                            }
                        }
#pragma unroll
                        for (int h = 0; h < 5; ++h) l[s][h] = (code == 4u || h == 4 || code == (uint32_t)h) ? lm : lx;
                    }
#pragma unroll
                    for (int h = 0; h < 5; ++h) words[h].v[k] = O::make(l[0][h], l[NS - 1][h]);
                    if (r < R) {
                        N[r] = O::make(0.f, 0.f);
                        D[r] = O::make(0.f, 0.f);
                    }
                }
#pragma unroll
                for (int h = 0; h < 5; ++h) tab[(h * Q + q) * 32 + lane] = words[h];
            }
            if constexpr (UNI) {
                wv[0] = O::uniform(O::make(w[0][0], w[NS - 1][0]));
            }
        }
        V eps = O::make(kEps, kEps);
        if constexpr (GCP) {
            eps = O::make(rd.eps[0], rd.eps[NS - 1]);
            if constexpr (UNI) eps = O::uniform(eps);
        }
        V wend;   // 1/n of the read's last position
        if constexpr (kDouble) wend = 1.0 / (double)gap(rd, 0, rd.L[0] - 1).d;
        else wend = O::make(link(rd, 0, rd.L[0]).w, link(rd, NS - 1, rd.L[NS - 1]).w);
        constexpr S kD0 = kDouble && !EXT ? (S)kTileD0 * (S)kScaled : (S)kTileD0;
        const V zero = O::make(0.f, 0.f), d0 = O::make(kD0, kD0);
        const bool first = u == 0;
        // the result lane adds the rows up to its pair's last step
        const int kres = u == NL - 1 ? H + G - 1 : -1;

        V Nl = zero;   // this lane's last N of the step before (the row T needs)
        V Ml = zero, Mul = zero, Iul = zero, Xul = first ? d0 : zero;
        // EXT: exponents of this lane, and of Ml, Mul, and Iul and Xul
        int e = 0, eMl = 0, eMul = 0, eIul = 0;
        bool empty = !first;
        sum.e = 0;
        int h = 4;
        uint32_t wcur = hap.codes(0);
        uint32_t wnext = hap.codes(1);
        RingRow fetched{};   // serial: row 32*b + t of the block of 32 rows after the next
        const RingRow* left = ring;      // rows of the column before this part
        RingRow* right = border;         // rows of its last column, one per step
        const bool writer = kParts && warp + 1 < parts && t == 31;
        if constexpr (SERIAL) {
            __syncwarp();
            if (warp > 0) {
                ring[t] = border[kBorderPad + t];   // a buffer has more than 96 rows
                fetched = border[kBorderPad + 32 + t];
            } else {
                ring[t] = ring[32 + t] = RingRow{zero, zero, d0, 0};
            }
            __syncwarp();
        }
        if constexpr (kBlockGroup) {
            // warp v writes ring v + 1 and reads ring v; ring 0 holds the boundary
            left = ring + warp * kRing;
            right = ring + (warp + 1) * kRing;
            if (warp == 0) ring[t] = ring[32 + t] = RingRow{zero, zero, d0, 0};
            __syncwarp();
        }
        auto four_steps = [&](int k0) {
            const uint32_t wpref = hap.codes((k0 >> 2) + 2);
            if constexpr (SERIAL) {
                if (warp > 0 && (k0 & 31) == 0) {
                    __syncwarp();
                    ring[(k0 + 32 + t) & (kRing - 1)] = fetched;
                    __syncwarp();
                    if (kBorderPad + 64 + (int64_t)k0 + t < rows) fetched = border[kBorderPad + 64 + k0 + t];
                }
            }
            V a4 = zero;
#pragma unroll kUnroll
            for (int s4 = 0; s4 < 4; ++s4) {
                const int k = k0 + s4;
                int hn = __shfl_up_sync(kFullMask, h, 1, G);
                if (t == 0) hn = (int)((wcur >> (8 * s4)) & 0xffu);
                h = hn;
                const Word* row = tab + h * (Q * 32) + lane;
                if constexpr (EXT) {
                    // lanes fill in the wavefront's first pass: centre the lane's scale on the
                    // first values it receives
                    if (k0 < G + 8 && empty && (Mul != 0.0 || Xul != 0.0 || Iul != 0.0)) {
                        const double xi = fmax(fabs(Xul), fabs(Iul));
                        e = Mul != 0.0 ? eMul - ilogb(fabs(Mul)) : eIul - ilogb(xi);
                        empty = false;
                    }
                    if (e - (eMul < eIul ? eMul : eIul) > kMaxShift) {
                        // a neighbour's values far above this lane's scale: coarsen the scale by
                        // an exact power of two first, so that the conversion cannot overflow;
                        // what falls out of range is negligible next to the incoming values
                        const int dM = Mul != 0.0 ? e - eMul : INT_MIN;
                        const int dI = (Xul != 0.0 || Iul != 0.0) ? e - eIul : INT_MIN;
                        const int over = (dM > dI ? dM : dI) - kMaxShift;
                        if (over > 0) {
                            const double f = over > 1022 ? 0.0 : pow2i(-over);
#pragma unroll
                            for (int r = 0; r < R; ++r) { N[r] *= f; D[r] *= f; }
                            Nl *= f;
                            if (k <= kres) sum.s[0] *= f;
                            e -= over;
                        }
                    }
                    const double fM = pow2i(e - eMul), fI = pow2i(e - eIul);
                    Mul *= fM;
                    Iul *= fI;
                    Xul *= fI;
                }
                // a position first forms what the next one takes from its old N, so that N is
                // replaced in place (with the old N carried along instead, the compiler moves
                // the lane's N by one register a step, on the FMA pipe)
                V P = O::fma(Mul, wv[0], Xul), I = O::fma(Iul, eps, Mul), X = zero, Ilast = zero;
                V Ic[SPAN], Xc[SPAN];   // I and X after position R-1-j
#pragma unroll
                for (int q = 0; q < Q; ++q) {
                    const Word lw = row[q * 32];
#pragma unroll
                    for (int i = 0; i < VN; ++i) {
                        const int r = q * VN + i;
                        if (r < R) {
                            if constexpr (UNI) X = O::add(D[r], I);
                            else X = O::fma(D[r], xv[r], I);
                            D[r] = O::fma(D[r], eps, N[r]);
                            const V Nnew = O::mul(lw.v[i], P);
                            Ilast = I;
                            if (r + 1 < R) {
                                P = O::fma(N[r], wv[UNI ? 0 : (r + 1 < R ? r + 1 : r)], X);
                                I = O::fma(I, eps, N[r]);
                            }
                            N[r] = Nnew;
                            if (r >= R - SPAN) {
                                Ic[R - 1 - r] = Ilast;
                                Xc[R - 1 - r] = X;
                            }
                        }
                    }
                }
                V Id = Ic[SPAN - 1], Xd = Xc[SPAN - 1], Ne = N[R - SPAN];
#pragma unroll
                for (int j = SPAN - 2; j >= 0; --j) {
                    Id = O::sel(holds[j], Ic[j], Id);
                    Xd = O::sel(holds[j], Xc[j], Xd);
                    Ne = O::sel(holds[j], N[R - 1 - j], Ne);
                }
                const V T = O::fma(Nl, wend, Id);
                if constexpr (kRowSums) {
                    if (k <= kres) sum.s[0] += (double)O::side(T, 0);
                } else {
                    if (k <= kres) a4 = O::add(a4, T);
                }
                Nl = Ne;
                if constexpr (kParts) {
                    // the last lane is at row k - 31; rows before the first land in the padding
                    // (serial) or in slots the next part has not reached yet.  serial: the row
                    // was fetched by this warp 64 steps ago or more
                    if (writer) right[SERIAL ? k + 1 : (k + 33) & (kRing - 1)] = RingRow{Nl, Id, Xd, e};
                }
                Mul = Ml;
                Ml = O::up(Nl, G);
                Iul = O::up(Id, G);
                Xul = O::up(Xd, G);
                if constexpr (EXT) {   // values travel with the sender's exponent
                    eMul = eMl;
                    eMl = __shfl_up_sync(kFullMask, e, 1, G);
                    eIul = eMl;
                }
                if constexpr (kParts) {
                    const RingRow b = left[(k + 1) & (kRing - 1)];  // broadcast
                    if (t == 0) {
                        Ml = b.n;
                        Iul = b.i;
                        Xul = b.x;
                        eMl = eIul = b.e;
                    }
                } else if (t == 0) {
                    Ml = zero;
                    Iul = zero;
                    Xul = d0;
                    eMl = eIul = 0;
                }
                if constexpr (EXT) {
                    // renormalise every 16 steps (exact powers of two); a value moves by at most
                    // 2^13 per row, so lanes stay within 2^300 of their scale meanwhile
                    if ((k & 15) == 15) {
                        double mx = fmax(k <= kres ? fabs(sum.s[0]) : 0.0, fmax(fabs(Id), fabs(Xd)));
#pragma unroll
                        for (int r = 0; r < R; ++r) mx = fmax(mx, fmax(fabs(N[r]), fabs(D[r])));
                        if (mx > 0.0) {
                            const int fe = ilogb(mx);
                            if (fe > 64 || fe < -64) {
                                const int kk = -fe < -1022 ? -1022 : (-fe > 1023 ? 1023 : -fe);
                                const double f = pow2i(kk);
#pragma unroll
                                for (int r = 0; r < R; ++r) { N[r] *= f; D[r] *= f; }
                                Nl *= f;
                                if (k <= kres) sum.s[0] *= f;
                                e += kk;
                            }
                        }
                    }
                    // past its last row a group's values are not the pair's and must not
                    // rescale the finished sum
                    if (k <= kres) sum.e = e;
                }
            }
            if constexpr (!kRowSums) {
                if (kres >= 0) {
#pragma unroll
                    for (int s = 0; s < NS; ++s) sum.s[s] += (double)O::side(a4, s);
                }
            }
            wcur = wnext;
            wnext = wpref;
        };
        if constexpr (!kBlockGroup) {
            if (SERIAL && warp > 0) {  // row 0, before the first step
                const RingRow r0 = left[0];
                if (t == 0) {
                    Ml = r0.n;
                    Iul = r0.i;
                    Xul = r0.x;
                    eMl = eIul = r0.e;
                }
            }
            for (int k0 = 0; k0 < K; k0 += 4) four_steps(k0);
        } else {
            const int nblk = (H + 32 + kBlock - 1) / kBlock;
            const int nsuper = nblk + kLag * (W - 1);
            for (int ss = 0; ss < nsuper; ++ss) {
                const int b = ss - kLag * warp;
                if (b >= 0 && b < nblk) {  // warp-uniform
                    if (b == 0 && warp > 0) {  // row 0, before the first step
                        const RingRow r0 = left[0];
                        if (t == 0) {
                            Ml = r0.n;
                            Iul = r0.i;
                            Xul = r0.x;
                            eMl = eIul = r0.e;
                        }
                    }
                    for (int k0 = b * kBlock; k0 < (b + 1) * kBlock; k0 += 4) four_steps(k0);
                }
                __syncthreads();
            }
        }
    }

    // All parts of a warp's task.  threshold: below half of it on a part's last column
    // a serial pair stops (0: never).  Returns false if it stopped.
    __device__ __forceinline__ static bool run(const Reads& rd, const Hap& hap, int H, int K, bool uni, Word* tab,
                                               RingRow* ring, RingRow* border, int64_t rows, int t, int warp, int lane,
                                               double threshold, Sum& sum, int parts = W) {
        if constexpr (!SERIAL) {
            if (uni) loop<true>(rd, hap, H, K, tab, ring, border, rows, t, warp, parts, lane, sum);
            else loop<false>(rd, hap, H, K, tab, ring, border, rows, t, warp, parts, lane, sum);
        } else {
            for (int part = 0; part < parts; ++part) {
                if (uni) loop<true>(rd, hap, H, K, tab, ring, border, rows, t, part, parts, lane, sum);
                else loop<false>(rd, hap, H, K, tab, ring, border, rows, t, part, parts, lane, sum);
                __syncwarp();   // the part's rows are written
                if (SPAN == 2 && threshold > 0.0 && part + 1 < parts) {
                    // M = N/n, I + D one row up = X on the part's last column
                    const int c = (part + 1) * 32 * (R - 1) + min_i((part + 1) * 32, rd.L[0] - G * parts * (R - 1));
                    const double inv_n = 1.0 / (double)gap(rd, 0, c).d;
                    double mass = 0.0;
                    for (int j = t; j <= H; j += 32) mass += (double)border[kBorderPad + j].n * inv_n + (double)border[kBorderPad + j].x;
#pragma unroll
                    for (int d = 16; d >= 1; d >>= 1) mass += __shfl_xor_sync(kFullMask, mass, d);
                    if (mass < 0.5 * threshold) return false;   // warp-uniform
                }
            }
        }
        return true;
    }
};

}  // namespace phmm
