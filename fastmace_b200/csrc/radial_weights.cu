// Per-edge radial weights W[e, path, channel] = hidden[e, :] . W4[:, path, channel] (the last layer of the radial MLP,
// fastmace/rewrites/generic/modules.py:454) or their d/dr, on the tensor cores.
//
// One persistent CTA per SM: 8 consumer warps (two groups of 128 threads, thread = channel = TMEM lane) and one warp that
// feeds the tensor cores. For a tile of edges the consumers split the 64 hidden radial features into tf32 value and
// remainder and write them as the N-side operand (K-major, 128-byte swizzle); then, path by path, bulk copies bring the
// path's 128 x 64 block of W4 (pre-split and pre-swizzled at packing time, 16 KB pieces) through a ring of stages, one
// thread issues the 3xTF32 MMAs (M = 128 channels, N = 256 edges, K = 64) into one of two TMEM accumulators, and the
// consumers store the path before.
//
// Every wait is bounded (tc::mbar_wait): if one gives up, the CTA raises FMB_STATUS_TENSOR_TIMEOUT, stops waiting
// everywhere, runs to its end and frees its tensor memory.

#include "stages.cuh"
#include "tc_common.cuh"
#include "generated/tp_generated.cuh"

namespace fmb {

namespace {

using namespace tc;

constexpr int kWeightThreads = 288;        // 8 consumer warps + the tensor-core warp
constexpr int kStageBytes = 16384;        // one (hi or lo) x (K half) piece of a path's weight block: 128 rows x 32
constexpr unsigned kSpin = 1u << 20;

// barrier slots
constexpr int kBarFull = 0, kBarEmpty = 8, kBarTFull = 16, kBarTEmpty = 18, kBarB = 20;

// State of the thread that feeds the tensor cores: it keeps the ring of weight pieces full (bulk copies, look-ahead
// of NST pieces across paths, rounds and work items: the sequence of pieces is periodic) and issues the MMAs of one
// path at a time. Counters wrap by comparison, there is no division on this thread's critical path.
template <int TN, int NST>
struct Feeder {
    uint32_t bar0, ring0, tmem_base, idesc;
    uint64_t desc_bh, desc_bl;
    const float* image;
    volatile int* abort_flag;
    uint32_t pieces;                  // 4 * paths: pieces of one pass over the weight image
    uint32_t total;                   // pieces this CTA consumes in all
    uint32_t step = 0, load = 0;      // pieces consumed / requested
    uint32_t st = 0, ph = 0;          // stage and parity of the next piece to consume
    uint32_t lst = 0, lph = 1;        // stage to refill and the parity its `empty` barrier has to show
    uint32_t piece = 0;               // next piece to request
    uint32_t gpath = 0, ground = 0;

    __device__ __forceinline__ uint32_t bar(int slot) const { return bar0 + 8u * (uint32_t)slot; }

    __device__ __forceinline__ void top_up() {
        while (load < total && load - step < (uint32_t)NST) {
            mbar_wait(bar(kBarEmpty) + 8u * lst, lph, abort_flag, kSpin);
            const uint32_t full = bar(kBarFull) + 8u * lst;
            mbar_expect_tx(full, kStageBytes);
            bulk_load(ring0 + lst * kStageBytes, image + (size_t)piece * (kStageBytes / 4), kStageBytes, full);
            ++load;
            if (++piece == pieces) piece = 0;
            if (++lst == (uint32_t)NST) { lst = 0; lph ^= 1u; }
        }
    }

    // waits until the consumers have staged the N-side operand of the next round
    __device__ __forceinline__ void begin_round() {
        top_up();
        mbar_wait(bar(kBarB), ground & 1u, abort_flag, kSpin);
        fence_after_sync();
        ++ground;
    }

    // the 24 MMAs of one path (3xTF32: weights_lo x hidden_hi, weights_hi x hidden_lo, weights_hi x hidden_hi, per K
    // half) into accumulator gpath & 1
    __device__ __forceinline__ void path() {
        const uint32_t buf = gpath & 1u;
        mbar_wait(bar(kBarTEmpty + buf), ((gpath >> 1) & 1u) ^ 1u, abort_flag, kSpin);
        fence_after_sync();
        const uint32_t d = tmem_base + buf * TN;
#pragma unroll
        for (int s4 = 0; s4 < 4; ++s4) {
            top_up();
            mbar_wait(bar(kBarFull) + 8u * st, ph, abort_flag, kSpin);
            fence_after_sync();
            const uint64_t adesc = make_desc(ring0 + st * kStageBytes);
            const int kh = s4 >> 1;
            if ((s4 & 1) == 0) {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    mma_tf32(d, adesc + (uint64_t)(2 * k), desc_bh + k_step<TN>(4 * kh + k), idesc, (s4 == 0 && k == 0) ? 0 : 1);
            } else {
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    mma_tf32(d, adesc + (uint64_t)(2 * k), desc_bl + k_step<TN>(4 * kh + k), idesc, 1);
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    mma_tf32(d, adesc + (uint64_t)(2 * k), desc_bh + k_step<TN>(4 * kh + k), idesc, 1);
            }
            mma_commit(bar(kBarEmpty) + 8u * st);
            ++step;
            if (++st == (uint32_t)NST) { st = 0; ph ^= 1u; }
        }
        mma_commit(bar(kBarTFull + buf));
        ++gpath;
    }
};

// Tiles of 256 consecutive edges; the consumers only move accumulator columns to global memory -- lane = channel, so a warp writes 128 contiguous bytes of
// one edge row per store (a path-major layout [path][edge][128], contiguous per tile, measured slower both for this
// kernel and for its readers). The hidden features of a tile are split and staged once for all paths, the accumulator of
// path p is stored while the tensor cores work on path p + 1 (or on the next tile's first). Bound by the stores: 4 * paths *
// 128 bytes per edge leave an SM at 25 bytes a cycle, 5,150 of the 5,400 cycles a path of 256 edges takes.
struct WeightArgs {
    const float* hidden;          // [edges][64]
    const float* image;           // fmb_layer_t.rad_img
    float* out;                   // [edges][n_paths * 128]
    const long long* limit;       // device scalar: rows at or beyond *limit - limit_offset are skipped
    long long limit_offset;
    int rows;                     // host bound on the rows of this launch
    uint32_t* error_word;
    const int32_t* row_index;     // or null: output row r comes from hidden row row_index[r]
};

constexpr int kWeightStages = 4;
constexpr int kWeightTile = 256;
constexpr int kWeightRing = 2 * kWeightTile * 256;                    // after the hi and lo N-side operands
constexpr int kWeightBars = kWeightRing + kWeightStages * kStageBytes;
constexpr int kWeightBytes = kWeightBars + 256 + 16 + 1024;

template <int P>
__global__ void __launch_bounds__(kWeightThreads, 1)
k_radial_weights(const __grid_constant__ WeightArgs a) {
    constexpr int TN = kWeightTile, NST = kWeightStages;
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    uint8_t* b_hi = smem;
    uint8_t* b_lo = smem + TN * 256;
    uint8_t* ring = smem + kWeightRing;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kWeightBars);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(smem + kWeightBars + 256);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(smem + kWeightBars + 260);
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](int slot) { return bar0 + 8u * (uint32_t)slot; };
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < NST; ++s) {
            mbar_init(bar(kBarFull + s), 1);
            mbar_init(bar(kBarEmpty + s), 1);
        }
        mbar_init(bar(kBarTFull), 1);
        mbar_init(bar(kBarTFull + 1), 1);
        mbar_init(bar(kBarTEmpty), 8);
        mbar_init(bar(kBarTEmpty + 1), 8);
        mbar_init(bar(kBarB), 8);
        *abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    if (warp == 8) tmem_alloc(smem_u32(tmem_slot), 2 * TN);
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = *tmem_slot;
    long long rows = a.rows;
    if (a.limit) rows = min(rows, max(*a.limit - a.limit_offset, 0LL));
    const int n_tiles = (int)((rows + TN - 1) / TN);

    if (warp == 8) {
        if (lane == 0) {
            Feeder<TN, NST> feed;
            feed.bar0 = bar0; feed.ring0 = smem_u32(ring); feed.tmem_base = tmem_base; feed.idesc = make_idesc<TN>();
            feed.desc_bh = make_desc(smem_u32(b_hi)); feed.desc_bl = make_desc(smem_u32(b_lo));
            feed.image = a.image; feed.abort_flag = abort_flag; feed.pieces = 4u * P;
            uint32_t total = 0;
            for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) total += 4u * P;
            feed.total = total;
            for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
                feed.begin_round();
                for (int p = 0; p < P; ++p) feed.path();
            }
        }
    } else {
        const int wg = tid >> 7, c = tid & 127, quadrant = warp & 3;
        const uint32_t lane_base = (uint32_t)(quadrant * 32) << 16;
        const int ld_row = warp * 8 + (lane & 7), ld_q = lane >> 3;
        constexpr int ld = P * kC;
        // the hidden features of the CTA's next tile are on their way while the last paths of this one are stored
        float4 held[TN / 64][4];
        auto fetch = [&](int t) {
#pragma unroll
            for (int sweep = 0; sweep < TN / 64; ++sweep) {
                const long long r = (long long)t * TN + ld_row + 64 * sweep;
                const bool ok = t < n_tiles && r < rows;
                const long long source = a.row_index ? (ok ? (long long)a.row_index[r] : 0) : r;
                const float4* src = reinterpret_cast<const float4*>(a.hidden + source * kRadial) + ld_q;
#pragma unroll
                for (int j = 0; j < 4; ++j) held[sweep][j] = ok ? __ldg(src + 4 * j) : make_float4(0.f, 0.f, 0.f, 0.f);
            }
        };
        auto stage = [&]() {
#pragma unroll
            for (int sweep = 0; sweep < TN / 64; ++sweep)
#pragma unroll
                for (int j = 0; j < 4; ++j) {
                    float4 hi, lo;
                    split_tf32(held[sweep][j], hi, lo);
                    const uint32_t off = tile_offset<TN>(ld_row + 64 * sweep, (ld_q + 4 * j) * 4);
                    *reinterpret_cast<float4*>(b_hi + off) = hi;
                    *reinterpret_cast<float4*>(b_lo + off) = lo;
                }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(kBarB));
        };
        uint32_t gpath = 0;
        fetch(blockIdx.x);
        if ((int)blockIdx.x < n_tiles) stage();
        for (int t = blockIdx.x; t < n_tiles; t += gridDim.x) {
            const long long e0 = (long long)t * TN;
            const long long eg = e0 + 128 * wg;                        // first edge of this group's 128 columns
            const int live = (int)min(128LL, max(rows - eg, 0LL));
            for (int p = 0; p < P; ++p) {
                const uint32_t buf = gpath & 1u;
                const uint32_t t0 = tmem_base + lane_base + buf * TN + 128u * (uint32_t)wg;
                if (p == P - 2) fetch(t + gridDim.x);
                mbar_wait(bar(kBarTFull + buf), (gpath >> 1) & 1u, abort_flag, kSpin);
                fence_after_sync();
                // the last path's MMAs are the last to read the operand: the next tile's replaces it before this path is
                // stored, so that the next tile's first MMAs run meanwhile
                if (p == P - 1 && t + (int)gridDim.x < n_tiles) stage();
                float* dst = a.out + eg * ld + p * kC + c;
                if (live == 128) {
#pragma unroll 1
                    for (int sb = 0; sb < 128; sb += 32, dst += 32 * ld) {
                        float w[16], v[16];
                        tmem_load_16x2(t0 + sb, t0 + sb + 16, w, v);
#pragma unroll
                        for (int q = 0; q < 16; ++q) dst[q * ld] = w[q];
#pragma unroll
                        for (int q = 0; q < 16; ++q) dst[(16 + q) * ld] = v[q];
                    }
                } else {
                    for (int sb = 0; sb < live; sb += 16) {
                        float w[16];
                        tmem_load<16>(t0 + sb, w);
#pragma unroll
                        for (int q = 0; q < 16; ++q)
                            if (sb + q < live) dst[(sb + q) * ld] = w[q];
                    }
                }
                fence_before_sync();
                __syncwarp();
                if (lane == 0) mbar_arrive(bar(kBarTEmpty + buf));
                ++gpath;
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 8) {
        __syncwarp();
        if (lane == 0 && *abort_flag && a.error_word) atomicOr(a.error_word, FMB_STATUS_TENSOR_TIMEOUT);
        tmem_free(tmem_base, 2 * TN);
    }
}

}  // namespace

namespace {

template <int P>
int launch_weights(const WeightArgs& a, int max_ctas, cudaStream_t stream) {
    static int sms = 0;
    FMB_CUDA_CHECK(opt_in_shared_memory((const void*)k_radial_weights<P>, kWeightBytes));
    if (sms == 0) {
        int dev = 0, count = 148;
        FMB_CUDA_CHECK(cudaGetDevice(&dev));
        FMB_CUDA_CHECK(cudaDeviceGetAttribute(&count, cudaDevAttrMultiProcessorCount, dev));
        sms = count;
    }
    const int tiles = (a.rows + kWeightTile - 1) / kWeightTile;
    const int ctas = max_ctas > 0 && max_ctas < sms ? max_ctas : sms;
    k_radial_weights<P><<<tiles < ctas ? tiles : ctas, kWeightThreads, kWeightBytes, stream>>>(a);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

}  // namespace

int radial_weights_tc(const float* hidden, const float* image, float* out, int rows, int n_paths, const long long* limit,
                      long long limit_offset, const int32_t* row_index, uint32_t* error_word, int max_ctas,
                      cudaStream_t stream) {
    if (!image) return FMB_ERR_UNSUPPORTED;
    if (rows <= 0) return FMB_OK;
    const WeightArgs a{hidden, image, out, limit, limit_offset, rows, error_word, row_index};
    switch (n_paths) {                       // a compile-time row length makes every store's offset an immediate
        case TpShape<0>::kPaths: return launch_weights<TpShape<0>::kPaths>(a, max_ctas, stream);
        case TpShape<1>::kPaths: return launch_weights<TpShape<1>::kPaths>(a, max_ctas, stream);
        case TpShape<2>::kPaths: return launch_weights<TpShape<2>::kPaths>(a, max_ctas, stream);
        default: return FMB_ERR_UNSUPPORTED;
    }
}

}  // namespace fmb
