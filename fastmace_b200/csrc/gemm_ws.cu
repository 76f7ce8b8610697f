// Warp-specialised tcgen05 / TMEM GEMM (3xTF32) for the per-irrep linears, the species skip and the first-layer
// fold: C[r, :] (+)= A[r, :] * W with strided rows (GemmArgs), N a multiple of 128 (of 64 where the image is padded), K a
// multiple of 32.
//
//   * The weights never pass through registers: their tf32 value / remainder parts are packed at load time into the
//     K-major 128-byte-swizzled operand layout and one thread brings the pieces in with bulk copies that complete on
//     an mbarrier.
//   * Eight loader warps bring the activation rows straight to their place in the operand tile (cp.async, four chunks
//     of 32 K in flight, so one round trip to memory per tile at K = 128) and split them there, value in place and
//     remainder beside it: a thread splits what it brought, so nothing but its own copies has to be waited for.
//   * The warp that issues the bulk copies issues the MMAs: per K = 8 the row values times [weight values | weight
//     remainders] (N = 2 TN in one instruction) and the row remainders times the weight values (N = TN) -- an MMA costs
//     about 60 cycles however narrow it is. It commits them to the stage's `empty` barrier; after the last chunk it
//     commits to the accumulator barrier and the loader warps turn into the epilogue (strided rows, accumulate, species
//     mask): the rows are turned through shared memory so that a store instruction writes whole row segments.
//   * Two accumulators in TMEM: value x value, and the two value x remainder products, added in the epilogue. The
//     tensor core truncates its accumulator at every instruction, so a sum that takes 3 K / 8 instructions into one
//     accumulator comes out 1.07e-6 of itself short at K = 128 (measured on positive operands); the remainder
//     products, 2^-11 of the total, lose nothing of weight in an accumulator of their own, and the K / 8 instructions
//     left leave a third of the bias.
//
// One CTA computes a 128 x TN tile of C; up to eight problems share a launch. A launch of few tiles is bound by the
// latency of one tile -- the bytes an SM pulls in (64 KB of rows and 1 KB of weights per column at K = 128), the split,
// the MMA chain, the epilogue -- and leaves most of the chip idle, so it is cut into narrower tiles: see
// gemm_ws_batch. Waits are bounded (tc::mbar_wait).

#include "gemm.cuh"
#include "tc_common.cuh"

#include <algorithm>

namespace fmb {

namespace {

using namespace tc;

constexpr int kWsThreads = 288;          // 8 loader / epilogue warps + the control warp
constexpr int kWsMaxStages = 4;
constexpr int kWsTK = 32;                // K elements per stage
constexpr int kWsPiece = 128 * kWsTK * 4;        // 16 KB: value or remainder part of 128 rows or columns of a K chunk
constexpr int kWsTail = 256 + 1024;
constexpr unsigned kWsSpin = 1u << 20;
constexpr int kWsMaxProblems = 8;

// a stage: A value, A remainder, W value, W remainder
constexpr int ws_stage_bytes(int tn) { return 2 * kWsPiece + 2 * tn * kWsTK * 4; }

struct WsRowMap {
    long long bs, rs;
    __device__ __forceinline__ long long operator()(int batch, int inner) const {
        return (long long)batch * bs + (long long)inner * rs;
    }
};

struct WsProblem {
    const float* a;
    const float* img;            // weight image: piece (n tile, k chunk) at float offset (nt * (k / 32) + kc) * 8192
    float* c;
    int m, n, k;
    int nm;                      // rows per batch, and 2^32 / nm rounded up (rows stay far below 2^32 / nm: exact quotients)
    uint32_t nm_magic;
    WsRowMap amap, cmap;
    int accumulate;
    const long long* m_limit;
    long long m_limit_offset;
    const int32_t* batch_species;
    int select;
    const int32_t* batch_list;   // optional: batch b of the rows is batch_list[b] (negative or >= batch_limit: no rows)
    int batch_limit;
    int tile_begin;              // first CTA of this problem
    int column_tiles;            // n / TN, and its magic number like nm's
    uint32_t column_magic;
};

struct WsBatch {
    WsProblem p[kWsMaxProblems];
    int count;
    uint32_t* error_word;
};

__device__ __forceinline__ void add_to_global(float* dst, const float4& v) {
    asm volatile("red.global.add.v4.f32 [%0], {%1, %2, %3, %4};" :: "l"(dst), "f"(v.x), "f"(v.y), "f"(v.z), "f"(v.w) : "memory");
}

// barrier slots: b_full[4], a_full[4], empty[4], acc
constexpr int kWsBFull = 0, kWsAFull = kWsMaxStages, kWsEmpty = 2 * kWsMaxStages, kWsAcc = 3 * kWsMaxStages;

__device__ __forceinline__ int quotient(int v, int divisor, uint32_t magic) {
    return divisor == 1 ? v : (int)__umulhi((uint32_t)v, magic);
}

__device__ __forceinline__ void copy_16(uint32_t dst, const float* src, bool live) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" :: "r"(dst), "l"(src), "r"(live ? 16 : 0) : "memory");
}

template <int TN, int STAGES>
__global__ void __launch_bounds__(kWsThreads, 1)
k_gemm_ws(const __grid_constant__ WsBatch batch) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr uint32_t kStageBytes = ws_stage_bytes(TN);
    constexpr uint32_t kWPart = TN * kWsTK * 4;              // bytes of one of the weight parts of a stage
    constexpr uint32_t kWHi = 2 * kWsPiece, kWLo = kWHi + kWPart;
    constexpr int stages = STAGES;
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + stages * kStageBytes);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + 3 * kWsMaxStages + 1);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t bar0 = smem_u32(bars);
    auto bar = [&](int slot) { return bar0 + 8u * (uint32_t)slot; };
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;

    int which = 0;
#pragma unroll
    for (int q = 1; q < kWsMaxProblems; ++q)
        if (q < batch.count && (int)blockIdx.x >= batch.p[q].tile_begin) which = q;
    // every field the loops use is copied to registers (the record is selected with a run-time index)
    const WsProblem& pr = batch.p[which];
    const float* __restrict__ a = pr.a;
    float* const c_out = pr.c;
    const WsRowMap amap = pr.amap, cmap = pr.cmap;
    const int accumulate = pr.accumulate, select = pr.select, k = pr.k, n = pr.n, nm = pr.nm, batch_limit = pr.batch_limit;
    const uint32_t nm_magic = pr.nm_magic;
    const int32_t* const batch_species = pr.batch_species;
    const int32_t* const batch_list = pr.batch_list;
    int m = pr.m;
    if (pr.m_limit) {
        const long long lim = *pr.m_limit - pr.m_limit_offset;
        if (lim < m) m = lim < 0 ? 0 : (int)lim;
    }
    const int local = blockIdx.x - pr.tile_begin, row_tile = quotient(local, pr.column_tiles, pr.column_magic);
    const int row0 = row_tile * 128, col0 = (local - row_tile * pr.column_tiles) * TN;
    if (row0 >= m) return;
    const int chunks = k / kWsTK;
    // row r is row `inner` of batch (atom) `b`; b < 0: the row is not written
    auto locate = [&](int r, int& b, int& inner) {
        const int q = quotient(r, nm, nm_magic);
        inner = r - q * nm;
        b = q;
        if (batch_list) {
            b = batch_list[q];
            if (b >= batch_limit) b = -1;
        }
        if (batch_species && b >= 0 && batch_species[b] != select) b = -1;
    };
    if (batch_list) {
        // the list is sorted by species, so most tiles hold none of this problem's rows
        int b = -1, inner;
        if (tid < 128 && row0 + tid < m) locate(row0 + tid, b, inner);
        if (!__syncthreads_or(b >= 0)) return;
    }

    // control warp: the weight piece of K chunk kc into its stage
    const uint32_t stage0 = smem_u32(smem);
    constexpr size_t kPieceFloats = 2 * kWsPiece / 4;          // [value 16 KB][remainder 16 KB] of one (128 columns, k chunk)
    // the tile's columns are a run of 8-row groups inside the pieces of its 128 columns
    const float* const pieces = pr.img + (size_t)(col0 >> 7) * chunks * kPieceFloats + (col0 & 127) * kWsTK;
    auto request = [&](int kc) {
        const int s = kc % stages;
        const uint32_t dst = stage0 + s * kStageBytes, full = bar(kWsBFull + s);
        const float* piece = pieces + (size_t)kc * kPieceFloats;
        if (elect_one()) {
            mbar_expect_tx(full, 2 * kWPart);
            bulk_load(dst + kWHi, piece, kWPart, full);
            bulk_load(dst + kWLo, piece + kWsPiece / 4, kWPart, full);
        }
        __syncwarp();
    };
    // loaders: thread t brings float4 (t & 7) of rows (t >> 3) + 32 i of a chunk; the 8 lanes that share a row read the
    // whole 128-byte line
    const int ld_row = tid >> 3, ld_q = tid & 7;
    const uint32_t own = tile_offset<128>(ld_row, ld_q * 4);         // its place in the tile; 32 rows further: + 4096 bytes
    const float* src[4];
    bool ok[4];
    auto fetch = [&](int kc) {
        const uint32_t dst = stage0 + (kc % stages) * kStageBytes + own;
#pragma unroll
        for (int i = 0; i < 4; ++i) copy_16(dst + i * 4096, src[i] + kc * kWsTK, ok[i]);
    };
    if (warp == 8) {
        if (elect_one()) {
#pragma unroll 1
            for (int s = 0; s < kWsMaxStages; ++s) {
                mbar_init(bar(kWsBFull + s), 1);
                mbar_init(bar(kWsAFull + s), 8);
                mbar_init(bar(kWsEmpty + s), 1);
            }
            mbar_init(bar(kWsAcc), 1);
            *abort_flag = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
        // the first weights travel during the rest of the set-up
#pragma unroll 1
        for (int kc = 0; kc < stages && kc < chunks; ++kc) request(kc);
    } else {
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const int row = row0 + ld_row + 32 * i;
            int b = -1, inner = 0;
            if (row < m) locate(row, b, inner);
            ok[i] = b >= 0;
            src[i] = a + (ok[i] ? amap(b, inner) : 0) + 4 * ld_q;
        }
#pragma unroll 1
        for (int kc = 0; kc < stages; ++kc) {
            if (kc < chunks) fetch(kc);
            asm volatile("cp.async.commit_group;" ::: "memory");
        }
        if (warp == 0) tmem_alloc(smem_u32(tmem_slot), 2 * TN);
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    if (warp == 8) {
        constexpr uint32_t idesc = make_idesc<TN>(), idesc_pair = make_idesc<2 * TN>();
#pragma unroll 1
        for (int kc = 0; kc < chunks; ++kc) {
            const int s = kc % stages;
            const uint32_t parity = (kc / stages) & 1;
            mbar_wait(bar(kWsBFull + s), parity, abort_flag, kWsSpin);
            mbar_wait(bar(kWsAFull + s), parity, abort_flag, kWsSpin);
            fence_after_sync();
            const uint32_t base = stage0 + s * kStageBytes;
            const uint64_t a_hi = make_desc(base), a_lo = make_desc(base + kWsPiece), w = make_desc(base + kWHi);
            const uint32_t go_on = kc > 0 ? 1 : 0;
            if (elect_one()) {
#pragma unroll
                for (int k8 = 0; k8 < 4; ++k8) {
                    // the stage's weight remainders follow its weight values, so one tile of 2 TN columns holds both
                    mma_tf32(tmem_base, a_hi + (uint64_t)(2 * k8), w + (uint64_t)(2 * k8), idesc_pair, k8 > 0 ? 1 : go_on);
                    mma_tf32(tmem_base + TN, a_lo + (uint64_t)(2 * k8), w + (uint64_t)(2 * k8), idesc, 1);
                }
                mma_commit(bar(kWsEmpty + s));
                if (kc == chunks - 1) mma_commit(bar(kWsAcc));
            }
            __syncwarp();
            // the stage of the chunk before is about to be free: refill it
            const int next = kc - 1 + stages;
            if (kc > 0 && next < chunks) {
                mbar_wait(bar(kWsEmpty + next % stages), ((next / stages) & 1) ^ 1, abort_flag, kWsSpin);
                request(next);
            }
        }
    } else {
        // ------------------------------------------------------------------ loaders
#pragma unroll 1
        for (int kc = 0; kc < chunks; ++kc) {
            // one group per chunk: all but the newest stages - 2 have arrived, chunk kc's among them
            asm volatile("cp.async.wait_group %0;" :: "n"(stages - 2) : "memory");
            const int s = kc % stages;
            uint8_t* const hi_tile = smem + s * kStageBytes + own;
            uint8_t* const lo_tile = hi_tile + kWsPiece;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float4 hi, lo;
                split_tf32(*reinterpret_cast<const float4*>(hi_tile + i * 4096), hi, lo);
                *reinterpret_cast<float4*>(hi_tile + i * 4096) = hi;
                *reinterpret_cast<float4*>(lo_tile + i * 4096) = lo;
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(kWsAFull + s));
            if (kc > 0) {
                const int next = kc - 1 + stages;                    // into the stage the MMAs of chunk kc - 1 give back
                if (next < chunks) {
                    mbar_wait(bar(kWsEmpty + next % stages), ((next / stages) & 1) ^ 1, abort_flag, kWsSpin);
                    fetch(next);
                }
                asm volatile("cp.async.commit_group;" ::: "memory");
            }
        }
        // ------------------------------------------------------------------ epilogue
        // Warps w and w + 4 read the same 32 accumulator lanes (= rows) and take half of the columns each. A row written
        // by its lane alone would make every store instruction touch 32 lines, so the warp's rows go through its
        // share of the first operand stage (free once the accumulator barrier has completed).
        constexpr int kCols = TN / 2, kSlots = kCols / 4;         // columns of a warp, float4 of a row
        const int quarter = warp & 3, half = warp >> 2;
        const int row_base = row0 + quarter * 32;
        long long my_row = -1;                                    // where this lane's row of C starts; negative: not written
        if (row_base + lane < m) {
            int b, inner;
            locate(row_base + lane, b, inner);
            if (b >= 0) my_row = cmap(b, inner);
        }
        float4* const turn = reinterpret_cast<float4*>(smem) + warp * 32 * kSlots;        // [32 rows][kSlots], XOR-swizzled
        mbar_wait(bar(kWsAcc), 0, abort_flag, kWsSpin);
        fence_after_sync();
#pragma unroll
        for (int col = 0; col < kCols; col += 16) {
            float v[16], u[16];
            const uint32_t taddr = tmem_base + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * kCols + col);
            tmem_load_16x2(taddr, taddr + TN, v, u);
#pragma unroll
            for (int q = 0; q < 4; ++q)
                turn[lane * kSlots + (((col >> 2) + q) ^ (lane & (kSlots - 1)))] =
                    make_float4(v[4 * q] + u[4 * q], v[4 * q + 1] + u[4 * q + 1], v[4 * q + 2] + u[4 * q + 2],
                                v[4 * q + 3] + u[4 * q + 3]);
        }
        __syncwarp();
        constexpr int kRowsPerStore = 32 / kSlots;
        const int slot = lane % kSlots;
        float* const c_tile = c_out + col0 + half * kCols + 4 * slot;
        const bool live = col0 + half * kCols < n;                    // the second half of the last tile may be padding
#pragma unroll 4
        for (int rr = lane / kSlots; rr < 32; rr += kRowsPerStore) {
            const float4 v = turn[rr * kSlots + (slot ^ (rr & (kSlots - 1)))];
            const long long row = __shfl_sync(0xffffffffu, my_row, rr);
            if (row >= 0 && live) {
                float* dst = c_tile + row;
                // accumulate: the add happens at the memory side (every element has one writer, so the sum is the
                // same old + new as a load and a store would give, without the round trip for the old values)
                if (accumulate) add_to_global(dst, v);
                else *reinterpret_cast<float4*>(dst) = v;
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        if (lane == 0 && *abort_flag && batch.error_word) atomicOr(batch.error_word, FMB_STATUS_TENSOR_TIMEOUT);
        tmem_free(tmem_base, 2 * TN);
    }
}

// ------------------------------------------------------------------------------------------------ many tiles
// A launch of more 128 x 128 tiles than the GPU has SMs: one persistent CTA per SM walks the tiles, so that nothing of
// a tile but its MMAs has to be waited for. Eight loader warps run up to two chunks ahead (into the next tile's), eight
// epilogue warps store a tile while the control warp's MMAs fill the other of two pairs of accumulators (value and
// remainder products of a tile: 2 x 256 TMEM columns). A tile by itself takes 11 k cycles (set-up 3 k, MMAs 3.1 k, epilogue
// 2.9 k, round trips); at one per SM a large launch is bound by those, here by the 3.1 k and by the 128 KB of rows that
// come from and go to memory.
constexpr int kWpThreads = 17 * 32;
constexpr int kWpStages = 3;
constexpr int kWpStageBytes = ws_stage_bytes(128);
constexpr int kWpTurnFloats = 32 * 32;                        // one epilogue warp: 32 rows of 32 columns
constexpr int kWpSmem = kWpStages * kWpStageBytes + 8 * kWpTurnFloats * 4 + kWsTail;
// barrier slots
constexpr int kWpBFull = 0, kWpAFull = kWpStages, kWpEmpty = 2 * kWpStages, kWpAccFull = 3 * kWpStages, kWpAccEmpty = kWpAccFull + 2;

// Where a warp is in the CTA's sequence of tiles: every role walks it with a cursor of its own. Tiles without a live row
// (the list of a species-dependent linear) are passed over.
struct TileCursor {
    int tile, total;
    const WsProblem* pr;
    int row0, col0, m, chunks;

    __device__ __forceinline__ void locate(int r, int& b, int& inner) const {
        const int q = quotient(r, pr->nm, pr->nm_magic);
        inner = r - q * pr->nm;
        b = q;
        if (pr->batch_list) {
            b = pr->batch_list[q];
            if (b >= pr->batch_limit) b = -1;
        }
        if (pr->batch_species && b >= 0 && pr->batch_species[b] != pr->select) b = -1;
    }

    // moves on to the first tile at or after `tile` that has rows to write; false: there is none
    __device__ __forceinline__ bool settle(const WsBatch& batch) {
        for (; tile < total; tile += gridDim.x) {
            int which = 0;
            for (int q = 1; q < batch.count; ++q)
                if (tile >= batch.p[q].tile_begin) which = q;
            pr = &batch.p[which];
            m = pr->m;
            if (pr->m_limit) {
                const long long lim = *pr->m_limit - pr->m_limit_offset;
                if (lim < m) m = lim < 0 ? 0 : (int)lim;
            }
            const int local = tile - pr->tile_begin, row_tile = quotient(local, pr->column_tiles, pr->column_magic);
            row0 = row_tile * 128;
            col0 = (local - row_tile * pr->column_tiles) * 128;
            chunks = pr->k / kWsTK;
            if (row0 >= m) continue;
            if (pr->batch_list) {
                bool any = false;
                for (int r = row0 + (int)(threadIdx.x & 31); r < row0 + 128 && r < m; r += 32) {
                    int b, inner;
                    locate(r, b, inner);
                    any = any || b >= 0;
                }
                if (!__any_sync(0xffffffffu, any)) continue;
            }
            return true;
        }
        return false;
    }
};

__global__ void __launch_bounds__(kWpThreads, 1)
k_gemm_walk(const __grid_constant__ WsBatch batch, int total) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    uint8_t* smem = smem_raw + ((1024u - (smem_u32(smem_raw) & 1023u)) & 1023u);
    constexpr uint32_t kWPart = 128 * kWsTK * 4, kWHi = 2 * kWsPiece;
    float4* const turn_all = reinterpret_cast<float4*>(smem + kWpStages * kWpStageBytes);
    uint64_t* bars = reinterpret_cast<uint64_t*>(smem + kWpStages * kWpStageBytes + 8 * kWpTurnFloats * 4);
    uint32_t* tmem_slot = reinterpret_cast<uint32_t*>(bars + kWpAccEmpty + 2);
    volatile int* abort_flag = reinterpret_cast<volatile int*>(tmem_slot + 1);
    const uint32_t bar0 = smem_u32(bars), stage0 = smem_u32(smem);
    auto bar = [&](int slot) { return bar0 + 8u * (uint32_t)slot; };
    const int tid = threadIdx.x, warp = uniform_warp(), lane = tid & 31;

    if (warp == 16) {
        if (elect_one()) {
#pragma unroll 1
            for (int s = 0; s < kWpStages; ++s) {
                mbar_init(bar(kWpBFull + s), 1);
                mbar_init(bar(kWpAFull + s), 8);
                mbar_init(bar(kWpEmpty + s), 1);
            }
            for (int s = 0; s < 2; ++s) {
                mbar_init(bar(kWpAccFull + s), 1);
                mbar_init(bar(kWpAccEmpty + s), 8);
            }
            *abort_flag = 0;
            asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        }
        __syncwarp();
    } else if (warp == 0) {
        tmem_alloc(smem_u32(tmem_slot), 512);
    }
    fence_before_sync();
    __syncthreads();
    fence_after_sync();
    const uint32_t tmem_base = __shfl_sync(0xffffffffu, *tmem_slot, 0);

    TileCursor cur{(int)blockIdx.x, total, nullptr, 0, 0, 0, 0};
    if (warp == 16) {
        // ------------------------------------------------------------------ control: weight copies and MMAs
        constexpr uint32_t idesc = make_idesc<128>(), idesc_pair = make_idesc<256>();
        TileCursor ahead = cur;
        int requested = 0, ahead_kc = 0;
        bool more = ahead.settle(batch);
        auto request = [&]() {
            if (!more) return;
            const int s = requested % kWpStages;
            mbar_wait(bar(kWpEmpty + s), ((requested / kWpStages) & 1) ^ 1, abort_flag, kWsSpin);
            const uint32_t dst = stage0 + s * kWpStageBytes + kWHi, full = bar(kWpBFull + s);
            const float* piece = ahead.pr->img + ((size_t)(ahead.col0 >> 7) * ahead.chunks + ahead_kc) * (2 * kWsPiece / 4);
            if (elect_one()) {
                mbar_expect_tx(full, 2 * kWPart);
                bulk_load(dst, piece, 2 * kWPart, full);
            }
            __syncwarp();
            ++requested;
            if (++ahead_kc == ahead.chunks) {
                ahead_kc = 0;
                ahead.tile += gridDim.x;
                more = ahead.settle(batch);
            }
        };
        for (int s = 0; s < kWpStages - 1; ++s) request();
        int done = 0;
        for (int turn = 0; cur.settle(batch); ++turn, cur.tile += gridDim.x) {
            const uint32_t acc = tmem_base + (uint32_t)(turn & 1) * 256u;
            mbar_wait(bar(kWpAccEmpty + (turn & 1)), ((turn >> 1) & 1) ^ 1, abort_flag, kWsSpin);
            fence_after_sync();
#pragma unroll 1
            for (int kc = 0; kc < cur.chunks; ++kc, ++done) {
                const int s = done % kWpStages;
                const uint32_t parity = (done / kWpStages) & 1;
                mbar_wait(bar(kWpBFull + s), parity, abort_flag, kWsSpin);
                mbar_wait(bar(kWpAFull + s), parity, abort_flag, kWsSpin);
                fence_after_sync();
                const uint32_t base = stage0 + s * kWpStageBytes;
                const uint64_t a_hi = make_desc(base), a_lo = make_desc(base + kWsPiece), w = make_desc(base + kWHi);
                const uint32_t go_on = kc > 0 ? 1 : 0;
                if (elect_one()) {
#pragma unroll
                    for (int k8 = 0; k8 < 4; ++k8) {
                        mma_tf32(acc, a_hi + (uint64_t)(2 * k8), w + (uint64_t)(2 * k8), idesc_pair, k8 > 0 ? 1 : go_on);
                        mma_tf32(acc + 128, a_lo + (uint64_t)(2 * k8), w + (uint64_t)(2 * k8), idesc, 1);
                    }
                    mma_commit(bar(kWpEmpty + s));
                    if (kc == cur.chunks - 1) mma_commit(bar(kWpAccFull + (turn & 1)));
                }
                __syncwarp();
                request();
            }
        }
    } else if (warp < 8) {
        // ------------------------------------------------------------------ loaders (as in k_gemm_ws)
        const int ld_row = tid >> 3, ld_q = tid & 7;
        const uint32_t own = tile_offset<128>(ld_row, ld_q * 4);
        const float* src[4];
        bool ok[4];
        int fetched = 0, kc = 0;
        auto place = [&]() {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                const int row = cur.row0 + ld_row + 32 * i;
                int b = -1, inner = 0;
                if (row < cur.m) cur.locate(row, b, inner);
                ok[i] = b >= 0;
                src[i] = cur.pr->a + (ok[i] ? cur.pr->amap(b, inner) : 0) + 4 * ld_q;
            }
        };
        bool more = cur.settle(batch);
        if (more) place();
        auto fetch = [&]() {
            if (more) {
                const int s = fetched % kWpStages;
                mbar_wait(bar(kWpEmpty + s), ((fetched / kWpStages) & 1) ^ 1, abort_flag, kWsSpin);
                const uint32_t dst = stage0 + s * kWpStageBytes + own;
#pragma unroll
                for (int i = 0; i < 4; ++i) copy_16(dst + i * 4096, src[i] + kc * kWsTK, ok[i]);
                ++fetched;
                if (++kc == cur.chunks) {
                    kc = 0;
                    cur.tile += gridDim.x;
                    more = cur.settle(batch);
                    if (more) place();
                }
            }
            asm volatile("cp.async.commit_group;" ::: "memory");
        };
        for (int s = 0; s < kWpStages - 1; ++s) fetch();
#pragma unroll 1
        for (int g = 0; g < fetched; ++g) {
            asm volatile("cp.async.wait_group %0;" :: "n"(kWpStages - 2) : "memory");
            const int s = g % kWpStages;
            uint8_t* const hi_tile = smem + s * kWpStageBytes + own;
            uint8_t* const lo_tile = hi_tile + kWsPiece;
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                float4 hi, lo;
                split_tf32(*reinterpret_cast<const float4*>(hi_tile + i * 4096), hi, lo);
                *reinterpret_cast<float4*>(hi_tile + i * 4096) = hi;
                *reinterpret_cast<float4*>(lo_tile + i * 4096) = lo;
            }
            fence_async_smem();
            __syncwarp();
            if (lane == 0) mbar_arrive(bar(kWpAFull + s));
            fetch();
        }
    } else {
        // ------------------------------------------------------------------ epilogue: warps w and w + 4 share 32 rows
        const int quarter = warp & 3, half = (warp >> 2) & 1;
        float4* const turn_buf = turn_all + (warp - 8) * (kWpTurnFloats / 4);      // [32 rows][8 float4], XOR-swizzled
        for (int turn = 0; cur.settle(batch); ++turn, cur.tile += gridDim.x) {
            const int row = cur.row0 + quarter * 32 + lane;
            long long my_row = -1;
            if (row < cur.m) {
                int b, inner;
                cur.locate(row, b, inner);
                if (b >= 0) my_row = cur.pr->cmap(b, inner);
            }
            const int accumulate = cur.pr->accumulate;
            float* const c_tile = cur.pr->c + cur.col0 + half * 64 + 4 * (lane & 7);
            const bool live = cur.col0 + half * 64 < cur.pr->n;       // the second half of the last tile may be padding
            mbar_wait(bar(kWpAccFull + (turn & 1)), (turn >> 1) & 1, abort_flag, kWsSpin);
            fence_after_sync();
            const uint32_t acc = tmem_base + (uint32_t)(turn & 1) * 256u + ((uint32_t)(quarter * 32) << 16) + (uint32_t)(half * 64);
#pragma unroll
            for (int part = 0; part < 2; ++part) {
#pragma unroll
                for (int col = 0; col < 32; col += 16) {
                    float v[16], u[16];
                    tmem_load_16x2(acc + part * 32 + col, acc + 128 + part * 32 + col, v, u);
#pragma unroll
                    for (int q = 0; q < 4; ++q)
                        turn_buf[lane * 8 + (((col >> 2) + q) ^ (lane & 7))] =
                            make_float4(v[4 * q] + u[4 * q], v[4 * q + 1] + u[4 * q + 1], v[4 * q + 2] + u[4 * q + 2],
                                        v[4 * q + 3] + u[4 * q + 3]);
                }
                __syncwarp();
                if (part == 1) {
                    fence_before_sync();
                    if (lane == 0) mbar_arrive(bar(kWpAccEmpty + (turn & 1)));
                }
#pragma unroll 4
                for (int rr = lane >> 3; rr < 32; rr += 4) {
                    const float4 v = turn_buf[rr * 8 + ((lane & 7) ^ (rr & 7))];
                    const long long at = __shfl_sync(0xffffffffu, my_row, rr);
                    if (at >= 0 && live) {
                        float* dst = c_tile + at + part * 32;
                        if (accumulate) add_to_global(dst, v);
                        else *reinterpret_cast<float4*>(dst) = v;
                    }
                }
                __syncwarp();
            }
        }
    }
    fence_before_sync();
    __syncthreads();
    if (warp == 0) {
        __syncwarp();
        if (lane == 0 && *abort_flag && batch.error_word) atomicOr(batch.error_word, FMB_STATUS_TENSOR_TIMEOUT);
        tmem_free(tmem_base, 512);
    }
}

// 2^32 / divisor, rounded up: __umulhi(v, magic) is v / divisor for v < 2^32 / divisor
uint32_t magic_of(int divisor) { return (uint32_t)(((1ull << 32) + (unsigned)divisor - 1) / (unsigned)divisor); }

template <int TN, int STAGES>
int launch_ws(const WsBatch& batch, int tiles, cudaStream_t stream) {
    constexpr int smem = STAGES * ws_stage_bytes(TN) + kWsTail;
    FMB_CUDA_CHECK(opt_in_shared_memory((const void*)k_gemm_ws<TN, STAGES>, smem));
    k_gemm_ws<TN, STAGES><<<tiles, kWsThreads, smem, stream>>>(batch);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

}  // namespace

int gemm_ws_batch(const GemmArgs* list, int count, cudaStream_t stream) {
    if (count < 1 || count > kWsMaxProblems) return FMB_ERR_UNSUPPORTED;
    WsBatch batch{};
    batch.count = count;
    batch.error_word = list[0].error_word;
    static const int sm_count = [] {
        int device = 0, sms = 148;
        if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        return sms;
    }();
    int tiles128 = 0;
    for (int q = 0; q < count; ++q) {
        const GemmArgs& g = list[q];
        const int columns = g.img_n > 0 ? g.img_n : g.n;             // whole column tiles of the image
        if (!g.b_img || columns % 128 != 0 || columns - g.n >= 128 || g.n % 64 != 0 || g.n > columns || g.k % kWsTK != 0 || g.k < kWsTK)
            return FMB_ERR_UNSUPPORTED;
        FMB_REQUIRE(g.a && g.c, "gemm_ws: null operand");
        FMB_REQUIRE(g.a_nm == g.c_nm, "gemm_ws: rows of A and C belong to the same batches");
        tiles128 += ceil_div(std::max(g.m, 0), 128) * (columns / 128);
    }
    // the widest tile that still gives every SM no more than one CTA when cut in four or two
    const int tn = tiles128 * 4 <= sm_count ? 32 : tiles128 * 2 <= sm_count ? 64 : 128;
    int tiles = 0;
    for (int q = 0; q < count; ++q) {
        const GemmArgs& g = list[q];
        WsProblem& p = batch.p[q];
        p.a = g.a; p.img = g.b_img; p.c = g.c;
        p.m = std::max(g.batch_list ? g.list_m : g.m, 0); p.n = g.n; p.k = g.k;
        p.nm = g.c_nm;
        p.nm_magic = g.c_nm > 1 ? magic_of(g.c_nm) : 0;
        p.amap = WsRowMap{g.a_bs, g.a_rs};
        p.cmap = WsRowMap{g.c_bs, g.c_rs};
        p.accumulate = g.accumulate;
        p.m_limit = g.m_limit; p.m_limit_offset = g.m_limit_offset;
        p.batch_species = g.batch_species; p.select = g.select;
        p.batch_list = g.batch_list; p.batch_limit = g.batch_limit;
        p.tile_begin = tiles;
        p.column_tiles = ceil_div(g.n, tn);
        p.column_magic = p.column_tiles > 1 ? magic_of(p.column_tiles) : 0;
        tiles += ceil_div(p.m, 128) * p.column_tiles;
    }
    if (tiles == 0) return FMB_OK;
    if (tn == 32) return launch_ws<32, 4>(batch, tiles, stream);
    if (tn == 64) return launch_ws<64, 4>(batch, tiles, stream);
    if (tiles <= sm_count) return launch_ws<128, 3>(batch, tiles, stream);
    FMB_CUDA_CHECK(opt_in_shared_memory((const void*)k_gemm_walk, kWpSmem));
    k_gemm_walk<<<sm_count, kWpThreads, kWpSmem, stream>>>(batch, tiles);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

}  // namespace fmb
