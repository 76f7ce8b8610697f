// Channelwise tensor product of the interactions after the first over a range of edges (the whole list, or a chunk of one
// too long for its radial weights to be held) whose radial weights are in memory, forward and per-edge adjoint: every per-edge operand streamed through shared memory, two channels per thread on
// the packed FP32 pipe (fma.rn.f32x2), the harmonics coupled once per edge.
//
// An edge's harmonics enter every channel in the same few combinations, T[path][m_out][m_in] = sum_me C Y[me]. The
// threads of a CTA compute them for a batch of edges at a time (a lane per coupling, from harmonics that a bulk copy
// brought) and read them back as broadcasts: per channel pair the forward pass is then 110
// packed FMAs for node l_max 1 and the adjoint 330, where coupling inside each thread took 126 + 86 scalar products and
// 456. In the adjoint the gradient of the weighted sender features serves dE/dx and the derivative of the weights, and
// the products of weighted features and message gradient are formed once for all the harmonics they couple to.
//
// Streaming: a group of 64 threads walks a contiguous range of edges; its first warp keeps STAGES - 1 edges ahead of the
// group with bulk copies that complete on mbarriers (weights, in the adjoint their d/dr, the sender's feature rows), a
// stage is handed back by one arrival per warp. Weights and rows are read from the stage where a path needs them and
// not copied to registers first, which is what lets node l_max 2 (71 message components) run in this form.
//
// Bound: the weights from HBM (4 P C bytes per edge and direction of the pass) for node l_max 0 and 1, the FMA pipe with
// two warps per scheduler for l_max 2 (860 packed FMAs, two cycles each, 255 registers); below a few hundred receivers the
// chain of a row's edges. Forward / adjoint with its gather, before (scalar or in-thread coupling) and after: 62 k
// edges of l_max 1 118 -> 75 and 250 -> 188 us; 748 k edges of l_max 2 2.29 -> 1.41 and 7.21 -> 4.43 ms; 88 k edges of
// l_max 0 92 -> 64 and 205 -> 135 us.
//
// On small and middle lists the chain of an edge counts (IPC 0.46 with the weights in L2 as well): requests by an elected
// lane of a uniform warp, couplings without divergence and one fold for all 17 sums took the adjoint / forward kernels of
// l_max 0 (88 k edges) from 105 to 90 and 59 to 47 us, of l_max 2 (98 k edges) from 491 to 454 and 181 to 178, the adjoint
// of l_max 1 (62 k edges) from 153 to 145; at 615 k edges of l_max 1 both are at the HBM (5.5 TB/s).

#include "stages.cuh"
#include "generated/tp_generated.cuh"
#include "generated/tp_coupled_generated.cuh"
#include "edge_gradient.cuh"
#include "fold.cuh"
#include "tc_common.cuh"

namespace fmb {

namespace {

constexpr int kGroup = kC / 2;                 // threads of a group: channels 2 c and 2 c + 1
constexpr unsigned kSpin = 1u << 20;

__device__ __forceinline__ void group_sync(int id) { asm volatile("bar.sync %0, %1;" :: "r"(id), "r"(kGroup) : "memory"); }

// What a group knows of a range of edges ahead of their use: the couplings of the next batch (Y and T double buffered, Y
// by bulk copy two batches ahead), and the senders and weight rows of the next two (four-byte asynchronous copies), so
// that the thread that requests an edge's rows never waits for an index.
template <int LIN, int BATCH>
struct Ahead {
    static constexpr int kT = TpCoupled<LIN>::kFloats;
    static constexpr int kFloats = 2 * BATCH * (kT + 16) + 8 * BATCH;
    static constexpr int kWarpEdges = BATCH / (kGroup / 32);         // a warp's share of a batch
    float* t;                                  // [2][BATCH][kT]
    float* y;                                  // [2][BATCH][16]
    int32_t* index;                            // [4][senders BATCH, weight rows BATCH]
    uint32_t bar;                              // two barriers
    const float* edge_sh;
    const int32_t* senders;
    const int32_t* slot;
    int w0;                                    // the edge whose weights are row 0 of tp_w
    int eb, ee;
    int c, sync_id;
    volatile int* abort_flag;

    __device__ __forceinline__ Ahead(float* memory, uint32_t bar_, const float* edge_sh_, const int32_t* senders_,
                                     const int32_t* slot_, int w0_, int eb_, int ee_, int c_, int sync_id_,
                                     volatile int* abort_)
        : t(memory), y(memory + 2 * BATCH * kT), index(reinterpret_cast<int32_t*>(memory + 2 * BATCH * (kT + 16))), bar(bar_),
          edge_sh(edge_sh_), senders(senders_), slot(slot_), w0(w0_), eb(eb_), ee(ee_), c(c_), sync_id(sync_id_), abort_flag(abort_) {}

    // thread c < BATCH: the indices of its edge of batch b
    __device__ __forceinline__ void look_up(int b) const {
        const int e = eb + b * BATCH + c;
        if (c < BATCH && e < ee) {
            const uint32_t dst = tc::smem_u32(index + (b & 3) * 2 * BATCH + c);
            asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(dst), "l"(senders + e) : "memory");
            if (slot) asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" :: "r"(dst + 4 * BATCH), "l"(slot + e) : "memory");
        }
    }
    __device__ __forceinline__ int sender(int e) const {
        const int k = e - eb;
        return index[((k / BATCH) & 3) * 2 * BATCH + k % BATCH];
    }
    // the row of tp_w that holds an edge's weights: its own, or with one row per pair of opposite edges the pair's
    __device__ __forceinline__ int weight_row(int e) const {
        const int k = e - eb;
        return slot ? index[((k / BATCH) & 3) * 2 * BATCH + BATCH + k % BATCH] : e - w0;
    }

    __device__ __forceinline__ void request(int b) const {
        const int first = eb + b * BATCH;
        if (c == 0 && first < ee) {
            const uint32_t bytes = (uint32_t)min(BATCH, ee - first) * 64u, full = bar + 8u * (b & 1);
            tc::mbar_expect_tx(full, bytes);
            tc::bulk_load(tc::smem_u32(y + (b & 1) * BATCH * 16), edge_sh + 16 * (long long)first, bytes, full);
        }
    }
    // the couplings of batch b: a lane per coupling, each warp half of the edges (with a run of couplings per thread the four
    // runs of a warp went one after the other: 350 cycles an edge of the 3,200 its chain takes)
    __device__ __forceinline__ void compute(int b) const {
        if (eb + b * BATCH >= ee) return;
        tc::mbar_wait(bar + 8u * (b & 1), (uint32_t)(b >> 1) & 1u, abort_flag, kSpin);
        const int first = (c >> 5) * kWarpEdges;
        const float* const from = y + ((b & 1) * BATCH + first) * 16;
        float* const to = t + ((b & 1) * BATCH + first) * kT;
#pragma unroll
        for (int k0 = 0; k0 < TpCoupled<LIN>::kEntries; k0 += 32) {
            const int k = k0 + (c & 31);
            if (k >= TpCoupled<LIN>::kEntries) break;
            const int4 term = __ldg(reinterpret_cast<const int4*>(TpCoupled<LIN>::terms()) + k);
            const float c0 = __int_as_float(term.x), c1 = __int_as_float(term.y);
            const float* const y0 = from + (term.z & 15);
            const float* const y1 = from + (term.z >> 8 & 15);
            float* const place = to + (term.z >> 16);
#pragma unroll
            for (int e = 0; e < kWarpEdges; ++e) place[e * kT] = fmaf(c1, y1[16 * e], c0 * y0[16 * e]);
        }
    }
    __device__ __forceinline__ void start() const {
        look_up(0);
        look_up(1);
        request(0);
        request(1);
        asm volatile("cp.async.wait_all;" ::: "memory");
        group_sync(sync_id);
    }
    // before the first edge of batch b: its couplings become visible and the indices of batch b + 1, and it is certain that
    // the harmonics of batch b and the couplings of batch b - 1 have been read
    __device__ __forceinline__ void enter(int b) const {
        asm volatile("cp.async.wait_all;" ::: "memory");
        group_sync(sync_id);
        look_up(b + 2);
        request(b + 2);
        compute(b + 1);
    }
    __device__ __forceinline__ const float4* row(int b, int el) const {
        return reinterpret_cast<const float4*>(t + ((b & 1) * BATCH + el) * kT);
    }
};

// One warp's requests for the edges' rows: all lanes wait and look the indices up, an elected one issues, so that the
// copies' operands stay in uniform registers (requests by a single thread took 850 cycles an edge, with the other warp
// waiting for it).
template <int LIN, int STAGES, bool TANGENT>
struct Rows {
    static constexpr int P = TpShape<LIN>::kPaths, IN = TpShape<LIN>::kInDim;
    static constexpr int kW = P * kC;
    static constexpr int kX = (TANGENT ? 2 : 1) * kW;           // float offset of the sender rows in a stage
    static constexpr int kStage = kX + IN * kC;
    float* ring;
    uint32_t bar;                              // full[STAGES], empty[STAGES]
    const float* tp_w;
    long long tangent_offset;
    const float* x;
    int ee, issued;
    volatile int* abort_flag;
    int stage = 0;
    uint32_t parity = 1;

    template <typename AheadT>
    __device__ __forceinline__ void issue(const AheadT& ahead) {
        tc::mbar_wait(bar + 8u * (STAGES + stage), parity, abort_flag, kSpin);
        const uint32_t full = bar + 8u * stage, dst = tc::smem_u32(ring) + stage * kStage * 4;
        const int weight_row = __shfl_sync(0xffffffffu, ahead.weight_row(issued), 0), sender = __shfl_sync(0xffffffffu, ahead.sender(issued), 0);
        const float* const w = tp_w + (long long)weight_row * kW;
        if (tc::elect_one()) {
            tc::mbar_expect_tx(full, kStage * 4);
            tc::bulk_load(dst, w, kW * 4, full);
            if (TANGENT) tc::bulk_load(dst + kW * 4, w + tangent_offset, kW * 4, full);
            tc::bulk_load(dst + kX * 4, x + (long long)sender * (IN * kC), IN * kC * 4, full);
        }
        __syncwarp();
        ++issued;
        if (++stage == STAGES) { stage = 0; parity ^= 1u; }
    }
};

// The receivers of the edges [e0, e1) of `total`: those whose row starts in the range (rows without edges among them, the
// trailing ones with the last range) and the one that straddles its beginning.
__device__ __forceinline__ void rows_of_range(const int32_t* __restrict__ row_ptr, int n_rows, long long e0, long long e1,
                                              long long total, int& first, int& last) {
    first = 0;
    last = n_rows;
    if (e0 > 0) {
        int lo = 0, hi = n_rows;
        while (lo < hi) {
            const int at = (lo + hi) >> 1;
            if (row_ptr[at + 1] > e0 || row_ptr[at] >= e0) hi = at; else lo = at + 1;
        }
        first = lo;
    }
    if (e1 < total) {
        int lo = first, hi = n_rows;
        while (lo < hi) {
            const int at = (lo + hi) >> 1;
            if (row_ptr[at] >= e1) hi = at; else lo = at + 1;
        }
        last = lo;
    }
}

template <int LIN, int STAGES, int BATCH>
constexpr int forward_group_floats() { return STAGES * Rows<LIN, STAGES, false>::kStage + Ahead<LIN, BATCH>::kFloats; }

// GROUPS = 1: a CTA owns a contiguous block of receivers. GROUPS > 1 (few receivers): a CTA owns one, its groups take
// runs of the row's edges and meet in shared memory at the end.
// RANGE: the launch covers [e0, e0 + e_span) of a list evaluated in chunks, else all of it (the extra state of a range
// costs the 128-register form 9 %).
template <int LIN, int STAGES, int BATCH, int GROUPS, int MINB, bool RANGE>
__global__ void __launch_bounds__(kGroup * GROUPS, MINB)
k_tp_forward_coupled(int n_rows, const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ senders,
                     const float* __restrict__ x, const float* __restrict__ edge_sh, const float* __restrict__ tp_w,
                     float* __restrict__ mid, uint32_t* __restrict__ error_word, const int32_t* __restrict__ slot,
                     long long e0, long long e_span) {
    constexpr int MID = TpShape<LIN>::kMidDim;
    extern __shared__ __align__(128) float smem[];
    __shared__ uint64_t bars[GROUPS * (2 * STAGES + 2)];
    __shared__ int abort_sh;
    const int uniform = tc::uniform_warp(), group = GROUPS > 1 ? uniform / (kGroup / 32) : 0, warp = uniform - group * (kGroup / 32);
    const int c = threadIdx.x - group * kGroup, lane = c & 31;
    int first = 0, last = n_rows, begin = 0, e1 = 0;
    if (RANGE) {
        const int total = row_ptr[n_rows];
        e1 = (int)min((long long)total, e0 + e_span);
        if (e0 > 0 && e0 >= total) return;
        begin = (int)e0;
        rows_of_range(row_ptr, n_rows, e0, e1, total, first, last);
    }
    const int r0 = first + (int)((long long)blockIdx.x * (last - first) / gridDim.x),
              r1 = first + (int)((long long)(blockIdx.x + 1) * (last - first) / gridDim.x);
    if (r0 >= r1) return;
    int eb = row_ptr[r0], ee = row_ptr[r1];
    if (RANGE) {
        eb = max(eb, begin);
        ee = min(ee, e1);
    }
    if (GROUPS > 1) {
        const int len = ee - eb;
        ee = eb + len * (group + 1) / GROUPS;
        eb = eb + len * group / GROUPS;
    }
    const uint32_t bar = tc::smem_u32(bars) + 8u * group * (2 * STAGES + 2);
    if (c == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(bar + 8 * s, 1);                            // full
            tc::mbar_init(bar + 8 * (STAGES + s), kGroup / 32);       // empty: one arrival per warp
        }
        tc::mbar_init(bar + 8 * (2 * STAGES), 1);
        tc::mbar_init(bar + 8 * (2 * STAGES + 1), 1);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    float* const own = smem + group * forward_group_floats<LIN, STAGES, BATCH>();
    float* const tail = own + STAGES * Rows<LIN, STAGES, false>::kStage;
    const Ahead<LIN, BATCH> ahead(tail, bar + 8 * (2 * STAGES), edge_sh, senders, slot, begin, eb, ee, c, 1 + group, &abort_sh);
    Rows<LIN, STAGES, false> rows{own, bar, tp_w, 0, x, ee, eb, &abort_sh};
    ahead.start();
    if (warp == 0)
        while (rows.issued < ee && rows.issued < eb + STAGES - 1) rows.issue(ahead);
    ahead.compute(0);
    int stage = 0, batch = -1, el = BATCH;
    uint32_t parity = 0;
    int e = eb;
    for (int i = r0; i < r1; ++i) {
        int re = GROUPS > 1 ? ee : row_ptr[i + 1];
        if (RANGE) re = min(re, e1);
        float2* const out = reinterpret_cast<float2*>(mid + ((long long)i * MID) * kC) + c;
        const bool begun = RANGE && row_ptr[i] < begin;                  // the range before holds the row's first edges
        float2 acc[MID];
#pragma unroll
        for (int k = 0; k < MID; ++k) acc[k] = begun ? out[(long long)k * (kC / 2)] : make_float2(0.0f, 0.0f);
#pragma unroll 1
        for (; e < re; ++e) {
            if (el == BATCH) {
                ahead.enter(++batch);
                el = 0;
            }
            if (warp == 0 && rows.issued < ee && rows.issued < e + STAGES) rows.issue(ahead);
            tc::mbar_wait(bar + 8 * stage, parity, &abort_sh, kSpin);
            const float* st = own + stage * Rows<LIN, STAGES, false>::kStage;
            tp_forward_coupled<LIN, kC / 2>(reinterpret_cast<const float2*>(st + Rows<LIN, STAGES, false>::kX) + c, ahead.row(batch, el),
                                    reinterpret_cast<const float2*>(st) + c, acc);
            __syncwarp();
            if (lane == 0) tc::mbar_arrive(bar + 8 * (STAGES + stage));
            if (++stage == STAGES) { stage = 0; parity ^= 1u; }
            ++el;
        }
        if (GROUPS == 1) {
#pragma unroll
            for (int k = 0; k < MID; ++k) out[(long long)k * (kC / 2)] = acc[k];
        } else {
            __syncthreads();                                          // every group is done with its stages
            float2* const part = reinterpret_cast<float2*>(smem);     // [GROUPS - 1][MID][64]
            if (group > 0) {
#pragma unroll
                for (int k = 0; k < MID; ++k) part[((group - 1) * MID + k) * kGroup + c] = acc[k];
            }
            __syncthreads();
            if (group == 0) {
#pragma unroll
                for (int k = 0; k < MID; ++k) {
                    float2 v = acc[k];
#pragma unroll
                    for (int q = 0; q < GROUPS - 1; ++q) {
                        const float2 o = part[(q * MID + k) * kGroup + c];
                        v.x += o.x;
                        v.y += o.y;
                    }
                    out[(long long)k * (kC / 2)] = v;
                }
            }
        }
    }
    __syncthreads();
    if (threadIdx.x == 0 && abort_sh && error_word) atomicOr(error_word, FMB_STATUS_TENSOR_TIMEOUT);
}

// Every CTA takes the same number of edges (an edge is independent of the others of its row). The gradients of the
// harmonics and of the length are summed over the channels by shuffles and across the two warps in shared memory, where a
// batch's edge-vector gradients are finished while the next batch is under way.
template <int LIN, int STAGES, int BATCH>
constexpr int adjoint_floats() { return STAGES * Rows<LIN, STAGES, true>::kStage + Ahead<LIN, BATCH>::kFloats; }

template <int LIN, int STAGES, int BATCH, int MINB>
__global__ void __launch_bounds__(kGroup, MINB)
k_tp_adjoint_coupled(int n_rows, const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ senders,
                     const float* __restrict__ x, const float* __restrict__ edge_sh, const float* __restrict__ edge_vec,
                     const float* __restrict__ tp_w, long long tangent_offset, const float* __restrict__ d_mid,
                     float* __restrict__ dxe, float4* __restrict__ qe, uint32_t* __restrict__ error_word,
                     const int32_t* __restrict__ slot, long long e0, long long e_span, long long dx0) {
    constexpr int IN = TpShape<LIN>::kInDim, MID = TpShape<LIN>::kMidDim;
    using RowsT = Rows<LIN, STAGES, true>;
    extern __shared__ __align__(128) float smem[];
    __shared__ uint64_t bars[2 * STAGES + 2];
    __shared__ int abort_sh, first_row_sh;
    __shared__ float red[2][BATCH][2][18];
    const int c = threadIdx.x, warp = tc::uniform_warp(), lane = c & 31;
    const long long total = min((long long)row_ptr[n_rows], e0 + e_span);
    if (e0 >= total) return;
    const int begin = (int)e0, e1 = (int)total, per_cta = (e1 - begin + (int)gridDim.x - 1) / (int)gridDim.x;
    const int eb = (int)min(total, begin + (long long)blockIdx.x * per_cta), ee = eb + min(e1 - eb, per_cta);
    if (eb >= ee) return;
    const uint32_t bar = tc::smem_u32(bars);
    if (c == 0) {
        for (int s = 0; s < STAGES; ++s) {
            tc::mbar_init(bar + 8 * s, 1);                            // full
            tc::mbar_init(bar + 8 * (STAGES + s), kGroup / 32);       // empty: one arrival per warp
        }
        tc::mbar_init(bar + 8 * (2 * STAGES), 1);
        tc::mbar_init(bar + 8 * (2 * STAGES + 1), 1);
        abort_sh = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncthreads();
    float* const tail = smem + STAGES * RowsT::kStage;
    const Ahead<LIN, BATCH> ahead(tail, bar + 8 * (2 * STAGES), edge_sh, senders, slot, begin, eb, ee, c, 1, &abort_sh);
    RowsT rows{smem, bar, tp_w, tangent_offset, x, ee, eb, &abort_sh};
    ahead.start();
    if (warp == 0) {
        while (rows.issued < ee && rows.issued < eb + STAGES - 1) rows.issue(ahead);
        int lo = 0, hi = n_rows - 1;
        while (lo < hi) {
            const int at = (lo + hi + 1) >> 1;
            if (row_ptr[at] <= eb) lo = at; else hi = at - 1;
        }
        if (lane == 0) first_row_sh = lo;
    }
    __syncthreads();
    int a = first_row_sh;
    int row_end = row_ptr[a + 1];
    float2 g[MID];
#pragma unroll
    for (int k = 0; k < MID; ++k) g[k] = __ldg(reinterpret_cast<const float2*>(d_mid + ((long long)a * MID + k) * kC) + c);
    ahead.compute(0);
    auto finish = [&](int b) {
        const int e = eb + b * BATCH + c;
        if (c >= BATCH || e >= ee) return;
        const float (&r)[2][18] = red[b & 1][c];
        float gy[16];
#pragma unroll
        for (int q = 0; q < 16; ++q) gy[q] = r[0][q] + r[1][q];
        const float4 uv = __ldg(reinterpret_cast<const float4*>(edge_vec) + e);
        float q3[3];
        edge_vector_gradient(gy, r[0][16] + r[1][16], uv.x, uv.y, uv.z, uv.w, q3);
        qe[e] = make_float4(q3[0], q3[1], q3[2], 0.0f);
    };
    int place;                                 // the sum that `fold` leaves in this lane
    {
        int id[17];
#pragma unroll
        for (int q = 0; q < 17; ++q) id[q] = q;
        fold_ids<17, 16>(id, lane);
        place = id[0];
    }
    int stage = 0, batch = -1, el = BATCH;
    uint32_t parity = 0;
#pragma unroll 1
    for (int e = eb; e < ee; ++e) {
        if (el == BATCH) {
            ahead.enter(++batch);
            el = 0;
            if (batch > 0) finish(batch - 1);
        }
        if (e >= row_end) {
            do { ++a; row_end = row_ptr[a + 1]; } while (e >= row_end);
#pragma unroll
            for (int k = 0; k < MID; ++k) g[k] = __ldg(reinterpret_cast<const float2*>(d_mid + ((long long)a * MID + k) * kC) + c);
        }
        if (warp == 0 && rows.issued < ee && rows.issued < e + STAGES) rows.issue(ahead);
        float2 dY2[16], dx[IN], dr2 = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < 16; ++q) dY2[q] = make_float2(0.0f, 0.0f);
#pragma unroll
        for (int q = 0; q < IN; ++q) dx[q] = make_float2(0.0f, 0.0f);
        tc::mbar_wait(bar + 8 * stage, parity, &abort_sh, kSpin);
        const float* st = smem + stage * RowsT::kStage;
        tp_backward_coupled<LIN, kC / 2>(reinterpret_cast<const float2*>(st + RowsT::kX) + c, ahead.row(batch, el),
                                 reinterpret_cast<const float2*>(st) + c, reinterpret_cast<const float2*>(st + RowsT::kW) + c, g, dY2,
                                 dr2, dx);
        __syncwarp();
        if (lane == 0) tc::mbar_arrive(bar + 8 * (STAGES + stage));
        if (++stage == STAGES) { stage = 0; parity ^= 1u; }
#pragma unroll
        for (int q = 0; q < IN; ++q) reinterpret_cast<float2*>(dxe + ((e - dx0) * IN + q) * kC)[c] = dx[q];
        // 16 + 1 sums over the channels: inside the warp here, the two warps meet in shared memory
        float sums[17];
#pragma unroll
        for (int q = 0; q < 16; ++q) sums[q] = dY2[q].x + dY2[q].y;
        sums[16] = dr2.x + dr2.y;
        fold<17, 16>(sums, lane);
        red[batch & 1][el][warp][place] = sums[0];
        ++el;
    }
    __syncthreads();
    finish(batch);
    if (c == 0 && abort_sh && error_word) atomicOr(error_word, FMB_STATUS_TENSOR_TIMEOUT);
}

// CTAs that fill the device once
int resident(const void* kernel, int threads, int smem) {
    int per_sm = 0, sms = 148, dev = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, (size_t)smem) != cudaSuccess || per_sm < 1) per_sm = 1;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    return per_sm * sms;
}

template <int LIN, int STAGES, int BATCH, int GROUPS, int MINB, bool RANGE = false>
int launch_forward(const TpArgs& t, cudaStream_t stream) {
    constexpr int smem = GROUPS * forward_group_floats<LIN, STAGES, BATCH>() * 4;
    auto kernel = k_tp_forward_coupled<LIN, STAGES, BATCH, GROUPS, MINB, RANGE>;
    FMB_CUDA_CHECK(opt_in_shared_memory((const void*)kernel, smem));
    static const int cap = resident((const void*)kernel, kGroup * GROUPS, smem);
    const int grid = GROUPS > 1 || t.n_rows < cap ? t.n_rows : cap;
    kernel<<<grid, kGroup * GROUPS, smem, stream>>>(t.n_rows, t.row_ptr, t.senders, t.x, t.edge_sh, t.tp_w, t.mid, t.error_word,
                                                    t.slot, t.chunk_e0, t.chunk_edges);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

template <int LIN, int STAGES, int BATCH, int MINB>
int launch_adjoint(const EdgeAdjointArgs& t, cudaStream_t stream) {
    constexpr int smem = adjoint_floats<LIN, STAGES, BATCH>() * 4;
    auto kernel = k_tp_adjoint_coupled<LIN, STAGES, BATCH, MINB>;
    FMB_CUDA_CHECK(opt_in_shared_memory((const void*)kernel, smem));
    static const int cap = resident((const void*)kernel, kGroup, smem);
    kernel<<<cap, kGroup, smem, stream>>>(t.n_rows, t.row_ptr, t.senders, t.x, t.edge_sh, t.edge_vec, t.tp_w, t.tangent_offset,
                                          t.d_mid, t.dxe, reinterpret_cast<float4*>(t.qe), t.error_word, t.slot, t.chunk_e0,
                                          t.chunk_edges, t.dx_e0);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

}  // namespace

int tp_forward_coupled_launch(const TpArgs& t, cudaStream_t stream) {
    // Few receivers leave SMs idle and a receiver's edges are a serial chain: four groups (two where the stages of node
    // l_max 2 do not fit four times) share a receiver while one CTA of that size per SM and two waves of them suffice.
    // 64 atoms: 31 -> 11 us (l_max 0); 249 atoms of 59 neighbours: 64 -> 31 us (l_max 1).
    const bool few = t.n_rows <= 296;
    // otherwise the shape (stages, batch, CTAs per SM) measured best: warps in flight count for more than stages. l_max 1,
    // 62 k edges: 75 us at 3 / 8 / 8, 86 at 3 / 16 / 6, 91 at 4 / 8 / 6; l_max 2, 748 k edges: 1.41 ms at 3 / 8 / 3, 1.46 at
    // 2 / 8 / 4, 1.70 at 3 / 4 / 4
    if (!t.whole_list) {
        if (t.lin == 0) return launch_forward<0, 6, 16, 1, 8, true>(t, stream);
        if (t.lin == 1) return launch_forward<1, 3, 8, 1, 7, true>(t, stream);
        if (t.lin == 2) return launch_forward<2, 3, 8, 1, 3, true>(t, stream);
    }
    if (t.lin == 0) return few ? launch_forward<0, 4, 16, 4, 1>(t, stream) : launch_forward<0, 6, 16, 1, 8>(t, stream);
    if (t.lin == 1) return few ? launch_forward<1, 4, 16, 4, 1>(t, stream) : launch_forward<1, 3, 8, 1, 8>(t, stream);
    if (t.lin == 2) return few ? launch_forward<2, 3, 8, 2, 1>(t, stream) : launch_forward<2, 3, 8, 1, 3>(t, stream);
    return FMB_ERR_UNSUPPORTED;
}

int tp_adjoint_coupled_launch(const EdgeAdjointArgs& t, cudaStream_t stream) {
    // shapes (stages, batch, CTAs per SM) measured with the gather behind them, 62 k edges of l_max 1: 188 us at 2 / 8 / 6,
    // 207 at 2 / 16 / 5, 208 at 3 / 8 / 5; 748 k edges of l_max 2: 4.43 ms at 2 / 4 / 4, 5.08 at 2 / 8 / 3, 5.55 at 3 / 4 / 3
    if (t.lin == 0) return launch_adjoint<0, 4, 16, 8>(t, stream);
    if (t.lin == 1) return launch_adjoint<1, 2, 8, 6>(t, stream);
    if (t.lin == 2) return launch_adjoint<2, 2, 4, 4>(t, stream);
    return FMB_ERR_UNSUPPORTED;
}

}  // namespace fmb
