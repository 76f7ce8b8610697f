// Channelwise tensor product of the interactions after the first with the last radial layer inside the kernel (node l_max
// 1): the per-edge radial weights and their d/dr are products of the tensor cores that never leave the SM, where the kernels of
// tp_coupled.cu read them from memory (per pair of edges and force call 8 P C bytes written and 24 P C read).
//
// The last radial layer stays in tensor memory. As fp16 values and remainders the columns of half the channels, 640 of them,
// take 320 of 512 TMEM columns as the first operand of the MMAs, K along the
// columns; two CTAs share a range of edges, one per half. An MMA whose first operand is in TMEM
// takes 12 cycles at N = 16 where one that reads 128 rows from shared memory takes 40 whatever its N. The second operand is the
// hidden radial features of a tile, split in the kernel: 16 edges, or 8 edges and their d/dr.
//
// A pair of fp16 numbers holds the 22 bits of a tf32 pair down to 2^-17 of the top of its scale. The features of an edge near
// the cutoff have a scale of their own (Splitter); the layer has one, and only layers whose products come out as the tf32
// pairs give them are packed (packing.onchip_is_accurate). Message and adjoint of single pairs against float64, relative
// to their norm: 1.2e-7 to 1.9e-7 at any length, 4e-7 with the weights of the tf32 pairs; with one scale for all lengths
// 8e-7 at 5.9 A, 1e-5 at 5.95 and 7e-3 at 5.99.
//
// Warps: eight that evaluate edges, each a contiguous range of its own, a lane two channels on the packed FP32 pipe (the
// bodies of tp_coupled.cu); four that carry a tile's weights from TMEM, where a lane is a channel of one path, to the
// edges' blocks in shared memory; two that split hidden features, one of which issues the MMAs; two that bring the senders'
// rows (16-byte asynchronous copies) and couple the harmonics. A tile is one edge (forward: two) of each of the eight
// ranges, so that a warp meets the edges of its rows one after the other. Registers are dealt again after the start.
// Every wait is bounded (tc::mbar_wait).
//
// Bound inside the SM, two evaluating warps per scheduler: adjoint / forward, 62 k edges, shared memory 66 / 63 %, FP32 pipe 58 /
// 33, issue slots 59 / 39, tensor pipe 19 / 16, HBM 14 / 4 % busy.
// Adjoint / forward kernel, streamed and here: 62 k edges 145 -> 160 and 72 -> 96 us, 615 k edges 1,378 -> 1,350 (1,595 with the
// gather behind it) and 650 -> 800, and no producers (2 x 43 us and 2 x 360 us on the second stream, which slowed what ran
// beside them): a step of 1,944 atoms 742 -> 666 us, a force call of 10,368 atoms 4,679 -> 3,825, one in chunks
// 6,190 -> 4,010.

#include "stages.cuh"
#include "generated/tp_generated.cuh"
#include "generated/tp_coupled_generated.cuh"
#include "fold.cuh"
#include "tc_common.cuh"

#include <cuda_fp16.h>

namespace fmb {

namespace {

using namespace tc;

constexpr unsigned kSpin = 1u << 20;
constexpr int kSlices = 2, kCh = kC / kSlices, kLanePairs = kCh / 2;
constexpr int kWorkers = 8;                    // evaluating warps
constexpr int kThreads = 512;
constexpr int kBSlots = 2;                     // tiles of hidden features between the split and the MMAs
constexpr int kBSlotBytes = 4096;              // [16 rows][64] fp16 values, then remainders
constexpr int kAccumulators = 2;
constexpr int kScaleSlots = 8;                 // tiles whose rows' scales are kept: tile k's are written while tile k - 4's may be read
constexpr float kNearest = 0.001953125f;       // A from the cutoff: closer edges are scaled like one there
constexpr int kHeader = 8;                     // floats before the weights
constexpr int kPartFloats = 20;                // of an edge's sums: 16 harmonics, the length, 3 unused

template <int LIN, bool ADJOINT>
struct Shape {
    static constexpr int P = TpShape<LIN>::kPaths, IN = TpShape<LIN>::kInDim, MID = TpShape<LIN>::kMidDim;
    static constexpr int kTiles = P / 2, kT = TpCoupled<LIN>::kFloats;
    static constexpr int kPerWorker = ADJOINT ? 1 : 2, kEdges = kWorkers * kPerWorker;          // of a tile
    static constexpr int kWColumns = 64 * kTiles, kDColumns = 16 * kTiles;
    // an edge's block of a stage (floats): weights, in the adjoint their d/dr, the sender's features, the couplings
    static constexpr int kW = P * kCh, kX = (ADJOINT ? 2 : 1) * kW, kCoupled = kX + IN * kCh, kBlock = kCoupled + kT;
    static constexpr int kStageBytes = kEdges * kBlock * 4;
    static constexpr int kStages = ADJOINT ? 4 : 3;
    static constexpr int kY = kEdges * 64;
    static constexpr int kWorkerRegisters = 168;                       // of 256 for a worker's and a feeding warp's thread together
    static constexpr int kB = 0, kStage0 = kBSlots * kBSlotBytes, kY0 = kStage0 + kStages * kStageBytes,
                         kScale0 = kY0 + kY, kBytes = kScale0 + kScaleSlots * 72 + 1024;
    static constexpr int kBFull = 0, kBEmpty = kBSlots, kDFull = 2 * kBSlots, kDEmpty = kDFull + kAccumulators,
                         kFull = kDEmpty + kAccumulators, kEmpty = kFull + kStages, kBars = kEmpty + kStages;
    static_assert(P % 2 == 0 && kWColumns + kAccumulators * kDColumns <= 512 && kBytes <= 226 * 1024 && kBlock % 4 == 0, "fits an SM");
};

struct OnChipArgs {
    int n_rows;
    const int32_t* row_ptr;
    const int32_t* senders;
    const float* x;
    const float* edge_sh;
    const float* edge_vec;
    const float* hidden;
    const float* tangent;
    const float* image;            // [kHeader] (packing.onchip_image), then [slice][tile][value, remainder][8][128][4] words
    float* mid;
    float* heads;                  // forward: [range][MID][C] sums of rows that begin in an earlier range
    int32_t* head_row;             // forward: [range] that row, or -1
    const float* d_mid;
    float* dxe;
    float* parts;                  // adjoint: [slice][part_stride][kPartFloats]
    long long part_stride;
    long long e0, e_span, dx0;
    uint32_t* error_word;
};

__device__ __forceinline__ void mma_f16_ts(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, int accumulate) {
    asm volatile(
        "{\n"
        ".reg .pred p;\n"
        "setp.ne.b32 p, %4, 0;\n"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n"
        "}\n"
        :: "r"(d), "r"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}

__device__ __forceinline__ void tmem_store_32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        :: "r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
           "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]), "r"(v[18]),
           "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]), "r"(v[27]), "r"(v[28]),
           "r"(v[29]), "r"(v[30]), "r"(v[31]) : "memory");
}

// the first row at or beyond which row_ptr reaches `target` (at most row_ptr[n]); one warp, 32 probes at a time
__device__ __forceinline__ int lower_row(const int32_t* __restrict__ row_ptr, int n, int target, int lane) {
    int lo = 0, hi = n;
    while (lo < hi) {
        const int at = lo + (int)((long long)(hi - lo) * lane / 32);
        const unsigned reached = __ballot_sync(0xffffffffu, row_ptr[at] >= target);
        const int first = reached ? __ffs(reached) - 1 : 32;
        const int below = __shfl_sync(0xffffffffu, at, first > 0 ? first - 1 : 0), above = __shfl_sync(0xffffffffu, at, first & 31);
        if (first < 32) hi = above;
        if (first > 0) lo = below + 1;
    }
    return lo;
}

// What every role knows of the CTA.
template <int LIN, bool ADJOINT>
struct Cta {
    using S = Shape<LIN, ADJOINT>;
    const OnChipArgs& a;
    uint8_t* smem;
    uint32_t bar0, tmem;
    volatile int* abort_flag;
    int slice, lane;
    int begin, until, share, range0;           // edges of the launch, edges of a range, the first worker's range

    __device__ __forceinline__ uint32_t bar(int slot) const { return bar0 + 8u * (uint32_t)slot; }
    __device__ __forceinline__ void wait(int slot, uint32_t parity) const { mbar_wait(bar(slot), parity, abort_flag, kSpin); }
    __device__ __forceinline__ void arrive(int slot) const {
        __syncwarp();
        if (lane == 0) mbar_arrive(bar(slot));
    }
    __device__ __forceinline__ int first(int worker) const {
        return (int)min((long long)until, begin + (long long)share * (range0 + worker));
    }
    // edge `q` of tile k, or -1: its range is through
    __device__ __forceinline__ int edge(int k, int q) const {
        const int at = k * S::kPerWorker + q % S::kPerWorker;
        const long long e = begin + (long long)share * (range0 + q / S::kPerWorker) + at;
        return at < share && e < until ? (int)e : -1;
    }
    __device__ __forceinline__ int tiles() const { return (first(1) - first(0) + S::kPerWorker - 1) / S::kPerWorker; }
    __device__ __forceinline__ float* scales(int k) const {
        return reinterpret_cast<float*>(smem + S::kScale0) + (k % kScaleSlots) * 16;
    }
    // per part of the split: whether a row of tile k may have a scale that is not 1
    __device__ __forceinline__ int* scaled(int k) const {
        return reinterpret_cast<int*>(smem + S::kScale0 + kScaleSlots * 64) + (k % kScaleSlots) * 2;
    }
    __device__ __forceinline__ float* block(int k, int q) const {
        return reinterpret_cast<float*>(smem + S::kStage0 + (k % S::kStages) * S::kStageBytes) + q * S::kBlock;
    }
};

// ------------------------------------------------------------------------------------------------ feeding warps

// exponent field of the power of two that brings v >= 0 to [1, 2), or as near as powers of two go
__device__ __forceinline__ unsigned power_below(float v) { return min(254u - (__float_as_uint(v) >> 23), 253u); }

// Hidden radial features into the second operand (16 rows of 64 fp16, K-major, 128-byte swizzle; values, then remainders): the
// 16 edges of a tile, or its 8 edges and then their d/dr. Two warps split 8 rows each, those of the next tile on their way
// meanwhile: a warp shares its scheduler with two that evaluate, and one for all 16 rows was what the adjoint waited for (615 k
// edges with the gather behind it, the scales below included: 1,788 -> 1,620 us).
//
// Features of an edge near the cutoff are a million times smaller than those of a bond: they vanish with the fourth power of
// its distance from the cutoff (envelope and Bessel functions), their d/dr with the third. fp16 numbers below 2^-14 are
// spaced 2^-24: a row whose largest magnitude is below 1/4 at the scale that all share would be held less exactly than by
// tf32 pairs (2^-23 of the largest). By those laws rows of edges of a certain length or more are brought up by a power
// of two, and what takes their products back is left in `scales`. (Looking for the largest magnitude of every row instead
// cost twice as much.)
template <int LIN, bool ADJOINT>
struct Splitter {
    using S = Shape<LIN, ADJOINT>;
    const Cta<LIN, ADJOINT>& c;
    const int part, col, half;                 // of the rows; of a row's 16 pieces of four; row of a pair
    const float* const from;
    const float scale, reach, cutoff, size;
    int apart, at, my_at;
    float length;
    float4 held[4];

    __device__ __forceinline__ Splitter(const Cta<LIN, ADJOINT>& c_, int part_)
        : c(c_), part(part_), col(c_.lane & 15), half(c_.lane >> 4), from((ADJOINT && part_ ? c_.a.tangent : c_.a.hidden) + 4 * (c_.lane & 15)),
          scale(__ldg(c_.a.image + (ADJOINT ? part_ : 0))), reach(__ldg(c_.a.image + 3)), cutoff(__ldg(c_.a.image + 4)),
          size(__ldg(c_.a.image + (ADJOINT && part_ ? 6 : 5))) {
        // row 2 i + half of this part is the edge at + i * apart; lane q < 8 looks at the length of its edge q
        const int range = c.range0 + (ADJOINT ? 0 : 4 * part), lane = c.lane;
        apart = (ADJOINT ? 2 : 1) * c.share;
        at = c.begin + c.share * (range + (ADJOINT ? half : 0)) + (ADJOINT ? 0 : half);
        my_at = c.begin + c.share * (range + (ADJOINT ? lane : lane >> 1)) + (ADJOINT ? 0 : lane & 1);
        fetch(0);
    }

    __device__ __forceinline__ void fetch(int k) {
        const int left = c.share - k * S::kPerWorker;          // edges of a range from this tile on
        const bool inside = ADJOINT || half < left;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int e = at + i * apart;
            held[i] = inside && (unsigned)e < (unsigned)c.until ? __ldg(reinterpret_cast<const float4*>(from + (long long)e * kRadial))
                                                                : make_float4(0.f, 0.f, 0.f, 0.f);
        }
        length = c.lane < 8 && (ADJOINT || (c.lane & 1) < left) && (unsigned)my_at < (unsigned)c.until
                     ? __ldg(c.a.edge_vec + 4ll * my_at + 3) : 0.0f;
        at += S::kPerWorker;
        my_at += S::kPerWorker;
    }

    __device__ __forceinline__ void put(int k, int tiles) {
        const bool small = !(length < reach);
        const unsigned near = __ballot_sync(0xffffffffu, small);
        if (near) {
            // power of two, as exponent field, for the row of this lane's edge if its largest is below 1/4 (4 law at most):
            // to [1, 8], so that features that are far above the law, by the rounding of what made them, still fit
            const float d = fmaxf(cutoff - length, kNearest), law = (ADJOINT && part ? d * d : d * d * d) * d * size;
            const unsigned field = small && law < 0.0625f ? power_below(law) : 127u;
            if (c.lane < 8) c.scales(k)[8 * part + c.lane] = __uint_as_float((254u - field) << 23);
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                if ((near >> 2 * i & 3u) == 0) continue;
                const float up = __uint_as_float(__shfl_sync(0xffffffffu, field, 2 * i + half) << 23);
                held[i].x *= up; held[i].y *= up; held[i].z *= up; held[i].w *= up;
            }
        }
        if (c.lane == 0) c.scaled(k)[part] = near != 0;
        uint2 value[4], rest[4];
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const float2 lo = make_float2(held[i].x * scale, held[i].y * scale), hi = make_float2(held[i].z * scale, held[i].w * scale);
            const __half2 vl = __float22half2_rn(lo), vh = __float22half2_rn(hi);
            const float2 bl = __half22float2(vl), bh = __half22float2(vh);
            const __half2 rl = __float22half2_rn(make_float2(lo.x - bl.x, lo.y - bl.y)),
                          rh = __float22half2_rn(make_float2(hi.x - bh.x, hi.y - bh.y));
            value[i] = make_uint2(reinterpret_cast<const uint32_t&>(vl), reinterpret_cast<const uint32_t&>(vh));
            rest[i] = make_uint2(reinterpret_cast<const uint32_t&>(rl), reinterpret_cast<const uint32_t&>(rh));
        }
        if (k + 1 < tiles) fetch(k + 1);
        const int slot = k % kBSlots;
        c.wait(S::kBEmpty + slot, ((uint32_t)(k / kBSlots) & 1u) ^ 1u);
        uint8_t* const tile = c.smem + S::kB + slot * kBSlotBytes + part * 1024;       // 8 rows
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = 2 * i + half, to = row * 128 + (((col >> 1) ^ row) << 4) + (col & 1) * 8;
            *reinterpret_cast<uint2*>(tile + to) = value[i];
            *reinterpret_cast<uint2*>(tile + 2048 + to) = rest[i];
        }
        fence_async_smem();
        c.arrive(S::kBFull + slot);
    }
};

// The first part of the split.
template <int LIN, bool ADJOINT>
__device__ __forceinline__ void split_features(const Cta<LIN, ADJOINT>& c) {
    const int tiles = c.tiles();
    Splitter<LIN, ADJOINT> split(c, 0);
#pragma unroll 1
    for (int k = 0; k < tiles; ++k) split.put(k, tiles);
}

// The MMAs of the tiles: remainder x value, value x remainder, value x value over K = 64, the small products first (the
// tensor core truncates its accumulator at every instruction); the second part of the next tile's split while they run.
template <int LIN, bool ADJOINT>
__device__ __forceinline__ void issue_products(const Cta<LIN, ADJOINT>& c) {
    using S = Shape<LIN, ADJOINT>;
    constexpr uint32_t idesc = (1u << 4) | ((uint32_t)(16 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);   // D fp32, A and B fp16
    const int tiles = c.tiles();
    Splitter<LIN, ADJOINT> split(c, 1);
    if (tiles > 0) split.put(0, tiles);
#pragma unroll 1
    for (int k = 0; k < tiles; ++k) {
        const int slot = k % kBSlots, acc = k % kAccumulators;
        c.wait(S::kBFull + slot, (uint32_t)(k / kBSlots) & 1u);
        c.wait(S::kDEmpty + acc, ((uint32_t)(k / kAccumulators) & 1u) ^ 1u);
        fence_after_sync();
        const uint64_t value = make_desc(smem_u32(c.smem + S::kB + slot * kBSlotBytes)), rest = value + (2048 >> 4);
        const uint32_t d = c.tmem + S::kWColumns + acc * S::kDColumns;
        if (elect_one()) {
#pragma unroll 1
            for (int j = 0; j < S::kTiles; ++j) {
                const uint32_t w = c.tmem + 64 * j;
#pragma unroll
                for (int s = 0; s < 4; ++s) mma_f16_ts(d + 16 * j, w + 32 + 8 * s, value + 2 * s, idesc, s > 0);
#pragma unroll
                for (int s = 0; s < 4; ++s) mma_f16_ts(d + 16 * j, w + 8 * s, rest + 2 * s, idesc, 1);
#pragma unroll
                for (int s = 0; s < 4; ++s) mma_f16_ts(d + 16 * j, w + 8 * s, value + 2 * s, idesc, 1);
            }
            mma_commit(c.bar(S::kBEmpty + slot));
            mma_commit(c.bar(S::kDFull + acc));
            mbar_arrive(c.bar(S::kDFull + acc));                      // hands on what the split left in `scales`
        }
        __syncwarp();
        if (k + 1 < tiles) split.put(k + 1, tiles);
    }
    // after a wait that ran out nobody may have waited for the last products: they end before tensor memory is given back
    if (*c.abort_flag && tiles > 0) {
        const int k = tiles - 1;
        for (unsigned spin = 0; spin < kSpin && !mbar_try(c.bar(S::kBEmpty + k % kBSlots), (uint32_t)(k / kBSlots) & 1u); ++spin) {}
    }
}

// eight columns of the accumulator back to the common scale
template <int FIRST>
__device__ __forceinline__ void unscale(float (&v)[16], const float4* scale) {
#pragma unroll
    for (int q = FIRST; q < FIRST + 8; q += 4) {
        const float4 s = scale[q / 4];
        const float2 a = __fmul2_rn(make_float2(v[q], v[q + 1]), make_float2(s.x, s.y)),
                     b = __fmul2_rn(make_float2(v[q + 2], v[q + 3]), make_float2(s.z, s.w));
        v[q] = a.x; v[q + 1] = a.y; v[q + 2] = b.x; v[q + 3] = b.y;
    }
}

// Weights of a tile from the accumulator (lane = channel of a path, column = edge) to the edges' blocks, at the common scale.
template <int LIN, bool ADJOINT>
__device__ __forceinline__ void carry_weights(const Cta<LIN, ADJOINT>& c, int quadrant) {
    using S = Shape<LIN, ADJOINT>;
    const int tiles = c.tiles(), at = (quadrant >> 1) * kCh + (quadrant & 1) * 32 + c.lane;
    const uint32_t base = c.tmem + ((uint32_t)(quadrant * 32) << 16) + S::kWColumns;
#pragma unroll 1
    for (int k = 0; k < tiles; ++k) {
        const int st = k % S::kStages, acc = k % kAccumulators;
        c.wait(S::kEmpty + st, ((uint32_t)(k / S::kStages) & 1u) ^ 1u);
        c.wait(S::kDFull + acc, (uint32_t)(k / kAccumulators) & 1u);
        fence_after_sync();
        // the scales of a part wait in registers in the adjoint (615 k edges 1,629 -> 1,595 us), in the forward pass in shared
        // memory (808 us, 821 in registers)
        const int2 scaled = *reinterpret_cast<const int2*>(c.scaled(k));
        const float4* const scales = reinterpret_cast<const float4*>(c.scales(k));
        float4 scale[4];
        if (ADJOINT && scaled.x) { scale[0] = scales[0]; scale[1] = scales[1]; }
        if (ADJOINT && scaled.y) { scale[2] = scales[2]; scale[3] = scales[3]; }
        float* const to = c.block(k, 0) + at;
#pragma unroll
        for (int j = 0; j < S::kTiles; ++j) {
            float v[16];
            tmem_load_16(base + acc * S::kDColumns + 16 * j, v);
            if (scaled.x) unscale<0>(v, ADJOINT ? scale : scales);
            if (scaled.y) unscale<8>(v, ADJOINT ? scale : scales);
            if (j == S::kTiles - 1) {
                fence_before_sync();
                c.arrive(S::kDEmpty + acc);
            }
#pragma unroll
            for (int q = 0; q < 16; ++q)
                to[(ADJOINT ? (q & 7) * S::kBlock + (q >> 3) * S::kW : q * S::kBlock) + 2 * j * kCh] = v[q];
        }
        c.arrive(S::kFull + st);
    }
}

// The senders' rows of this half of the channels and the couplings of half a tile's edges; indices and harmonics a tile ahead.
template <int LIN, bool ADJOINT>
__device__ __forceinline__ void bring_rows(const Cta<LIN, ADJOINT>& c, int part) {
    using S = Shape<LIN, ADJOINT>;
    constexpr int N = S::kEdges / 2, kEntries = TpCoupled<LIN>::kEntries, kPerLane = (kEntries + 31) / 32;
    const int lane = c.lane, tiles = c.tiles(), q0 = part * N;
    const float scale = __ldg(c.a.image + 2);
    float c0[kPerLane], c1[kPerLane];
    int at[kPerLane];
#pragma unroll
    for (int j = 0; j < kPerLane; ++j) {
        const int4 term = __ldg(reinterpret_cast<const int4*>(TpCoupled<LIN>::terms()) + min(lane + 32 * j, kEntries - 1));
        c0[j] = __int_as_float(term.x) * scale;
        c1[j] = __int_as_float(term.y) * scale;
        at[j] = term.z;
    }
    float* const y = reinterpret_cast<float*>(c.smem + S::kY0) + q0 * 16;
    const float* const from = c.a.x + c.slice * kCh + (lane >> 4) * kC + 4 * (lane & 15);
    int sender = 0;
    float4 harmonics = make_float4(0.f, 0.f, 0.f, 0.f);
    auto fetch = [&](int k) {
        if (lane < N) {
            const int e = c.edge(k, q0 + lane);
            sender = e >= 0 ? __ldg(c.a.senders + e) : 0;
        }
        if (lane < 4 * N) {
            const int e = c.edge(k, q0 + (lane >> 2));
            harmonics = e >= 0 ? __ldg(reinterpret_cast<const float4*>(c.a.edge_sh + 16 * (long long)e) + (lane & 3))
                               : make_float4(0.f, 0.f, 0.f, 0.f);
        }
    };
    fetch(0);
#pragma unroll 1
    for (int k = 0; k < tiles; ++k) {
        const int st = k % S::kStages;
        c.wait(S::kEmpty + st, ((uint32_t)(k / S::kStages) & 1u) ^ 1u);
        // half a warp per component: 16 pieces of 16 bytes
        float* const first = c.block(k, q0);
        const uint32_t dst = smem_u32(first + S::kX) + 16 * lane;
#pragma unroll
        for (int j = 0; j < N * S::IN / 2; ++j) {
            const int q = 2 * j / S::IN, component = 2 * j % S::IN;
            const int s = __shfl_sync(0xffffffffu, sender, q);
            const float* src = from + (long long)s * (S::IN * kC) + component * kC;
            const uint32_t to = dst + (q * S::kBlock + component * kCh) * 4;
            asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(to), "l"(src) : "memory");
        }
        asm volatile("cp.async.mbarrier.arrive.noinc.shared.b64 [%0];" :: "r"(c.bar(S::kFull + st)) : "memory");
        if (lane < 4 * N) reinterpret_cast<float4*>(y)[lane] = harmonics;
        __syncwarp();
        if (k + 1 < tiles) fetch(k + 1);
#pragma unroll
        for (int j = 0; j < kPerLane; ++j) {
            if (lane + 32 * j < kEntries) {
                float* const to = first + S::kCoupled + (at[j] >> 16);
                const float* const y0 = y + (at[j] & 15);
                const float* const y1 = y + (at[j] >> 8 & 15);
#pragma unroll
                for (int q = 0; q < N; ++q) to[q * S::kBlock] = fmaf(c1[j], y1[16 * q], c0[j] * y0[16 * q]);
            }
        }
        c.arrive(S::kFull + st);
    }
    asm volatile("cp.async.wait_all;" ::: "memory");                  // in flight still only after a wait that ran out
}

// ------------------------------------------------------------------------------------------------ evaluating warps

// The rows with edges in this warp's range: the first may have begun in an earlier one (its sum goes to `heads` and is added to
// the row afterwards). Rows without edges are passed over by a search: k_finish_rows writes them, spread over the GPU. (With
// them written here 20,000 isolated atoms behind a crystal of 2,744 were one warp's: 7,660 us a force call.)
template <int LIN>
__device__ __forceinline__ void forward_range(const Cta<LIN, false>& c, int worker) {
    using S = Shape<LIN, false>;
    const int lane = c.lane, range = c.range0 + worker, first = c.first(worker), end = c.first(worker + 1), tiles = c.tiles();
    int row = first < end ? lower_row(c.a.row_ptr, c.a.n_rows, first + 1, lane) - 1 : 0, row_end = 0, k = 0;
    const bool head = first < end && __ldg(c.a.row_ptr + row) < first;
    if (c.slice == 0 && lane == 0) c.a.head_row[range] = head ? row : -1;
    float* to = c.a.heads + (long long)range * S::MID * kC;
    for (int e = first; e < end; ++row) {
        row_end = __ldg(c.a.row_ptr + row + 1);
        if (row_end <= e) {
            row = lower_row(c.a.row_ptr, c.a.n_rows, e + 1, lane) - 1;
            row_end = __ldg(c.a.row_ptr + row + 1);
        }
        if (!head || e > first) to = c.a.mid + (long long)row * S::MID * kC;
        const int re = min(row_end, end);
        float2 acc[S::MID];
#pragma unroll
        for (int q = 0; q < S::MID; ++q) acc[q] = make_float2(0.0f, 0.0f);
#pragma unroll 1
        for (; e < re; ++e) {
            const int odd = (e - first) & 1, st = k % S::kStages;
            if (!odd) c.wait(S::kFull + st, (uint32_t)(k / S::kStages) & 1u);
            const float* const from = c.block(k, 2 * worker + odd);
            tp_forward_coupled<LIN, kLanePairs>(reinterpret_cast<const float2*>(from + S::kX) + lane,
                                                reinterpret_cast<const float4*>(from + S::kCoupled),
                                                reinterpret_cast<const float2*>(from) + lane, acc);
            if (odd || e + 1 == end) {
                c.arrive(S::kEmpty + st);
                ++k;
            }
        }
        float2* const out = reinterpret_cast<float2*>(to + c.slice * kCh) + lane;
#pragma unroll
        for (int q = 0; q < S::MID; ++q) out[q * (kC / 2)] = acc[q];
    }
    for (; k < tiles; ++k) {                                             // the others' tiles
        c.wait(S::kFull + k % S::kStages, (uint32_t)(k / S::kStages) & 1u);
        c.arrive(S::kEmpty + k % S::kStages);
    }
}

// The range's edges: gradients of the senders' features and, summed over this half of the channels, of the harmonics and the
// length.
template <int LIN>
__device__ __forceinline__ void adjoint_range(const Cta<LIN, true>& c, int worker) {
    using S = Shape<LIN, true>;
    const int lane = c.lane, first = c.first(worker), end = c.first(worker + 1), tiles = c.tiles();
    constexpr int kHalf = 9;                   // of 17 sums, behind the first step of `fold`
    const float inverse = __ldg(c.a.image + 2), dr_scale = __ldg(c.a.image) / __ldg(c.a.image + 1);
    int place;                                 // the sum that `fold` leaves in this lane
    {
        int id[17];
#pragma unroll
        for (int q = 0; q < 17; ++q) id[q] = q;
        fold_ids<17, 16>(id, lane);
        place = id[0];
    }
    const float factor = place == 16 ? dr_scale : inverse;
    const float2* const g_from = reinterpret_cast<const float2*>(c.a.d_mid + c.slice * kCh) + lane;
    float2* dx_to = reinterpret_cast<float2*>(c.a.dxe + (first - c.a.dx0) * (S::IN * kC) + c.slice * kCh) + lane;
    float* part_to = c.a.parts + (c.slice * c.a.part_stride + first - 1) * kPartFloats + place;      // of the edge before
    int row = first < end ? max(lower_row(c.a.row_ptr, c.a.n_rows, first + 1, lane) - 1, 0) - 1 : 0, row_end = first;
    float2 g[S::MID];
#pragma unroll
    for (int q = 0; q < S::MID; ++q) g[q] = make_float2(0.0f, 0.0f);
    // the edge before: its sums over half the warp, the rest of which is added up beside the next edge's products
    float sums[17];
#pragma unroll
    for (int q = 0; q < 17; ++q) sums[q] = 0.0f;
    int k = 0;
#pragma unroll 1
    for (int e = first; e < end; ++e, ++k) {
        const int st = k % S::kStages;
        if (e >= row_end) {
            do { ++row; row_end = __ldg(c.a.row_ptr + row + 1); } while (e >= row_end);
#pragma unroll
            for (int q = 0; q < S::MID; ++q) g[q] = __ldg(g_from + ((long long)row * S::MID + q) * (kC / 2));
        }
        float2 dY2[16], dx[S::IN], dr2 = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < 16; ++q) dY2[q] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < S::IN; ++q) dx[q] = make_float2(0.0f, 0.0f);
        c.wait(S::kFull + st, (uint32_t)(k / S::kStages) & 1u);
        const float* const from = c.block(k, worker);
        fold<kHalf, 8>(sums, lane);
        if (e > first) *part_to = sums[0] * factor;
        part_to += kPartFloats;
        tp_backward_coupled<LIN, kLanePairs>(reinterpret_cast<const float2*>(from + S::kX) + lane,
                                             reinterpret_cast<const float4*>(from + S::kCoupled),
                                             reinterpret_cast<const float2*>(from) + lane,
                                             reinterpret_cast<const float2*>(from + S::kW) + lane, g, dY2, dr2, dx);
        c.arrive(S::kEmpty + st);
#pragma unroll
        for (int q = 0; q < S::IN; ++q) dx_to[q * (kC / 2)] = dx[q];
        dx_to += S::IN * (kC / 2);
#pragma unroll
        for (int q = 0; q < 16; ++q) sums[q] = dY2[q].x + dY2[q].y;
        sums[16] = dr2.x + dr2.y;
        fold_step<17, 16>(sums, lane);
    }
    if (first < end) {
        fold<kHalf, 8>(sums, lane);
        *part_to = sums[0] * factor;
    }
    for (; k < tiles; ++k) {                                             // the others' tiles
        c.wait(S::kFull + k % S::kStages, (uint32_t)(k / S::kStages) & 1u);
        c.arrive(S::kEmpty + k % S::kStages);
    }
}

template <int LIN, bool ADJOINT>
__global__ void __launch_bounds__(kThreads, 1)
k_tp_onchip(const __grid_constant__ OnChipArgs a) {
    using S = Shape<LIN, ADJOINT>;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    __shared__ uint64_t bars[S::kBars];
    __shared__ uint32_t tmem_slot;
    __shared__ int abort_sh;
    uint8_t* const smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    const int warp = uniform_warp(), lane = threadIdx.x & 31;
    const int total = a.row_ptr[a.n_rows];
    const int begin = ADJOINT ? (int)min((long long)total, a.e0) : 0, until = ADJOINT ? (int)min((long long)total, a.e0 + a.e_span) : total;
    const int ranges = (int)(gridDim.x / kSlices) * kWorkers;
    if (warp == 12) {
        if (elect_one()) {
            for (int q = 0; q < kBSlots; ++q) {
                mbar_init(smem_u32(bars + S::kBFull + q), 2);             // the two parts of the split
                mbar_init(smem_u32(bars + S::kBEmpty + q), 1);
            }
            for (int q = 0; q < kAccumulators; ++q) {
                mbar_init(smem_u32(bars + S::kDFull + q), 2);             // the products, and their issuer
                mbar_init(smem_u32(bars + S::kDEmpty + q), 4);
            }
            for (int q = 0; q < S::kStages; ++q) {
                mbar_init(smem_u32(bars + S::kFull + q), 4 + 2 * 33);     // weights, rows (a copy per lane), couplings
                mbar_init(smem_u32(bars + S::kEmpty + q), kWorkers);
            }
            abort_sh = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        tmem_alloc(smem_u32(&tmem_slot), 512);
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const Cta<LIN, ADJOINT> c{a, smem, smem_u32(bars), __shfl_sync(0xffffffffu, tmem_slot, 0), &abort_sh, (int)(blockIdx.x % kSlices), lane,
                              begin, until, (until - begin + ranges - 1) / ranges, (int)(blockIdx.x / kSlices) * kWorkers};
    if (warp < 8) {
        // this half of the last radial layer into tensor memory: lane = row, 32 words of value pairs, 32 of remainders
        const uint4* const image = reinterpret_cast<const uint4*>(a.image + kHeader) + (size_t)c.slice * S::kTiles * 2 * 1024 + (warp & 3) * 32 + lane;
        for (int part = warp >> 2; part < 2 * S::kTiles; part += 2) {
            uint32_t v[32];
#pragma unroll
            for (int q = 0; q < 8; ++q) {
                const uint4 u = __ldg(image + part * 1024 + q * 128);
                v[4 * q] = u.x; v[4 * q + 1] = u.y; v[4 * q + 2] = u.z; v[4 * q + 3] = u.w;
            }
            tmem_store_32(c.tmem + ((uint32_t)((warp & 3) * 32) << 16) + 32 * part, v);
        }
        asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    // the two halves of the CTA share the 512 x 128 registers of the launch
    if (warp < 8) {
        asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" :: "n"(S::kWorkerRegisters));
        if constexpr (ADJOINT) adjoint_range<LIN>(c, warp);
        else forward_range<LIN>(c, warp);
    } else {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" :: "n"(256 - S::kWorkerRegisters));
        if (warp < 12) carry_weights(c, warp & 3);
        else if (warp == 12) issue_products(c);
        else if (warp == 13) split_features(c);
        else bring_rows(c, warp - 14);
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 12) {
        if (lane == 0 && abort_sh && a.error_word) atomicOr(a.error_word, FMB_STATUS_TENSOR_TIMEOUT);
        __syncwarp();
        tmem_free(c.tmem, 512);
    }
}

// Zeroes the rows without edges (a lane looks at a row, a warp writes) and adds the sums of the ranges behind a row's first to the
// row, in order: one CTA per range, the first of a row does it.
constexpr int kFinishThreads = 512;
__global__ void __launch_bounds__(kFinishThreads)
k_finish_rows(int n_rows, int ranges, int row_floats, const int32_t* __restrict__ row_ptr, const float* __restrict__ heads,
              const int32_t* __restrict__ head_row, float* __restrict__ mid) {
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    for (int base = (warp * gridDim.x + blockIdx.x) * 32; base < n_rows; base += gridDim.x * kFinishThreads) {
        const int mine = base + lane;
        unsigned empty = __ballot_sync(0xffffffffu, mine < n_rows && __ldg(row_ptr + mine) == __ldg(row_ptr + mine + 1));
        for (; empty; empty &= empty - 1) {
            float4* const to = reinterpret_cast<float4*>(mid + (long long)(base + __ffs(empty) - 1) * row_floats);
            for (int q = lane; q < row_floats / 4; q += 32) to[q] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);
        }
    }
    const int range = blockIdx.x, row = head_row[range];
    if (row < 0 || (range > 0 && head_row[range - 1] == row)) return;
    for (int q = threadIdx.x; q < row_floats / 4; q += kFinishThreads) {
        float4* const to = reinterpret_cast<float4*>(mid + (long long)row * row_floats) + q;
        float4 sum = *to;
        for (int r = range; r < ranges && head_row[r] == row; ++r) {
            const float4 v = __ldg(reinterpret_cast<const float4*>(heads + (long long)r * row_floats) + q);
            sum.x += v.x; sum.y += v.y; sum.z += v.z; sum.w += v.w;
        }
        *to = sum;
    }
}

int device_sms() {
    static const int sms = [] {
        int dev = 0, count = 148;
        if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev);
        return count;
    }();
    return sms;
}

template <int LIN, bool ADJOINT>
int launch(const OnChipArgs& a, cudaStream_t stream) {
    using S = Shape<LIN, ADJOINT>;
    FMB_CUDA_CHECK(opt_in_shared_memory((const void*)k_tp_onchip<LIN, ADJOINT>, S::kBytes));
    const int grid = device_sms() / kSlices * kSlices, ranges = grid / kSlices * kWorkers;
    k_tp_onchip<LIN, ADJOINT><<<grid, kThreads, S::kBytes, stream>>>(a);
    FMB_LAUNCH_CHECK();
    if (!ADJOINT) {
        k_finish_rows<<<ranges, kFinishThreads, 0, stream>>>(a.n_rows, ranges, S::MID * kC, a.row_ptr, a.heads, a.head_row, a.mid);
        FMB_LAUNCH_CHECK();
    }
    return FMB_OK;
}

}  // namespace

long long tp_onchip_scratch_floats(int lin, long long edges) {
    // node l_max 0 has four paths of one component and too little to do per edge: 142 + 75 us for the adjoint and the forward
    // kernel of 88 k edges, 90 + 47 in tp_coupled.cu
    if (lin != 1) return -1;
    const long long ranges = device_sms() / kSlices * kWorkers;
    const long long forward = ranges * (TpShape<1>::kMidDim * kC + 1), adjoint = kSlices * edges * kPartFloats;
    return forward > adjoint ? forward : adjoint;
}

int tp_forward_onchip(const TpOnChipArgs& t, cudaStream_t stream) {
    if (t.lin != 1) return FMB_ERR_UNSUPPORTED;
    OnChipArgs a{};
    a.n_rows = t.n_rows; a.row_ptr = t.row_ptr; a.senders = t.senders; a.x = t.x; a.edge_sh = t.edge_sh; a.edge_vec = t.edge_vec; a.hidden = t.hidden;
    a.image = t.image; a.mid = t.mid; a.heads = t.scratch; a.error_word = t.error_word;
    a.head_row = reinterpret_cast<int32_t*>(t.scratch + (long long)(device_sms() / kSlices * kWorkers) * TpShape<1>::kMidDim * kC);
    return launch<1, false>(a, stream);
}

int tp_adjoint_onchip(const TpOnChipArgs& t, cudaStream_t stream) {
    if (t.lin != 1) return FMB_ERR_UNSUPPORTED;
    OnChipArgs a{};
    a.n_rows = t.n_rows; a.row_ptr = t.row_ptr; a.senders = t.senders; a.x = t.x; a.edge_sh = t.edge_sh; a.edge_vec = t.edge_vec; a.hidden = t.hidden;
    a.tangent = t.tangent; a.image = t.image; a.d_mid = t.d_mid; a.dxe = t.dxe; a.parts = t.scratch; a.part_stride = t.part_stride;
    a.e0 = t.e0; a.e_span = t.e_span; a.dx0 = t.dx0; a.error_word = t.error_word;
    return launch<1, true>(a, stream);
}

}  // namespace fmb
