// Adjoint of the interactions with per-edge hand-over instead of the mirror evaluation (buffers for the whole list where
// they fit, for one chunk of it otherwise).
//
// The mirror kernels (interaction.cu) make every receiver's CTA evaluate each of its edges twice -- as stored and in
// the opposite direction -- because that yields the sender-side gradient and the force without a scatter; the price is
// the gather of the mirror receiver's whole message-gradient row (20 KB per edge for the medium model), which makes
// that kernel L2-bandwidth bound. Here every directed edge is evaluated once, in its receiver's row, and hands over
//   * the gradient of its sender's features  dxe[e] = dE/dx_sender from this edge   ([IN][128] floats), and
//   * the gradient of its edge vector        qe[e]  = dE/dv_e                        (3 floats),
// and two light gather kernels finish the job through the mirror map e -> e' (the edge sender(e) <- receiver(e) with
// the opposite image; it exists because the neighbour list is full):
//   dE/dx_a = sum over the row of a of dxe[e'],      F_a = -(sum over the row of qe[e] - qe[e']),
//   virial_a = sum over the row of v_e (x) qe[e].
// Everything is summed in a fixed order; there are no atomics. Per edge the L2 traffic drops from 37 KB to about 14 KB
// and the coupling arithmetic halves.
//
// Replaces autograd through conv_tp + scatter_sum (fastmace/rewrites/generic/modules.py:485-486) like the mirror
// kernels; the reference's own edge-owned kernel scatters with atomicAdd (factorized_projected.cuh:258-353).

#include "stages.cuh"
#include "edge_gradient.cuh"
#include "tc_common.cuh"
#include "generated/tp_generated.cuh"

#include <cstdlib>

namespace fmb {

namespace {

template <int LIN, bool FLIP, bool NEED_DX> struct TpBackwardSel;
#define FMB_TP_BACKWARD_SEL(LIN_)                                                                                      \
    template <bool FLIP, bool NEED_DX> struct TpBackwardSel<LIN_, FLIP, NEED_DX> {                                     \
        template <typename... A> static __device__ __forceinline__ void run(A&&... a) {                               \
            tp_backward_##LIN_<FLIP, NEED_DX>(a...);                                                                   \
        }                                                                                                              \
    };
FMB_TP_BACKWARD_SEL(0)
FMB_TP_BACKWARD_SEL(1)
FMB_TP_BACKWARD_SEL(2)

constexpr int kBatch = 8;

// mirror[e] = index of the edge (sender = receiver(e), receiver = sender(e), image = -image(e)), or -1. With `slot`:
// the edges below *listed_below that stand for their pair (no opposite edge, or the lower index of the two) are listed
// in `list`; they and their opposite edges get the position as their slot (the order of the list depends on the atomics; the slots are only
// names of rows).
__global__ void k_mirror(const long long* __restrict__ count_ptr, int capacity, const int32_t* __restrict__ edge_index,
                         const float* __restrict__ unit_shifts, const int32_t* __restrict__ row_ptr,
                         int32_t* __restrict__ mirror, uint32_t* __restrict__ status,
                         const long long* __restrict__ listed_below, int32_t* __restrict__ slot,
                         int32_t* __restrict__ list, unsigned long long* __restrict__ list_count, int list_capacity) {
    const long long count = *count_ptr;
    const long long listed = slot ? *listed_below : 0;
    for (long long e = (long long)blockIdx.x * blockDim.x + threadIdx.x; e < count; e += (long long)gridDim.x * blockDim.x) {
        const int s = edge_index[e], r = edge_index[capacity + e];
        const float u0 = -unit_shifts[3 * e], u1 = -unit_shifts[3 * e + 1], u2 = -unit_shifts[3 * e + 2];
        // row s is sorted by (sender, image): first entry whose sender is >= r
        int lo = row_ptr[s], hi = row_ptr[s + 1];
        const int end = hi;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (edge_index[mid] < r) lo = mid + 1; else hi = mid;
        }
        int found = -1;
        for (int q = lo; q < end && edge_index[q] == r; ++q) {
            if (unit_shifts[3 * q] == u0 && unit_shifts[3 * q + 1] == u1 && unit_shifts[3 * q + 2] == u2) {
                found = q;
                break;
            }
        }
        mirror[e] = found;
        if (found < 0) atomicOr(status, FMB_STATUS_NO_MIRROR);
        if (slot && e < listed && (found < 0 || e < found)) {
            const unsigned long long k = atomicAdd(list_count, 1ull);
            if (k < (unsigned long long)list_capacity) {
                slot[e] = (int)k;
                if (found >= 0) slot[found] = (int)k;
                list[k] = (int)e;
            } else {
                slot[e] = 0;                                   // a row that exists; the status word says it is wrong
                if (found >= 0) slot[found] = 0;
                atomicOr(status, FMB_STATUS_PAIR_OVERFLOW);
            }
        }
    }
}

// Per-edge adjoint of the tensor product: CTA per receiver, thread per channel.
template <int LIN, int MINB>
__global__ void __launch_bounds__(kC, MINB)
k_tp_adjoint_edges(int n_atoms, int n_rows, int n_valid, long long chunk_e0, long long chunk_edges,
                   const long long* __restrict__ count_ptr, const int32_t* __restrict__ row_ptr,
                   const int32_t* __restrict__ senders, const float* __restrict__ x, const float* __restrict__ edge_sh,
                   const float* __restrict__ edge_vec, const float* __restrict__ tp_w, long long tangent_offset,
                   const float* __restrict__ d_mid, float* __restrict__ dxe, float4* __restrict__ qe, long long dx0) {
    constexpr int P = TpShape<LIN>::kPaths, IN = TpShape<LIN>::kInDim, MID = TpShape<LIN>::kMidDim;
    __shared__ float red[kBatch][4][18];
    const int c = threadIdx.x, warp = c >> 5, lane = c & 31;
    // this launch covers the edges [e0, e1) (a chunk of the list: tp_w holds their weights); a row that straddles two
    // chunks is simply visited by both, every edge is independent
    const long long count = *count_ptr;
    const long long e0 = chunk_e0, e1 = min(count, chunk_e0 + chunk_edges);
    if (e0 >= e1) return;
    int first = 0;
    if (e0 > 0) {
        int lo = 0, hi = n_atoms;
        while (lo < hi) {
            const int mid = (lo + hi) >> 1;
            if (row_ptr[mid + 1] > e0) hi = mid; else lo = mid + 1;
        }
        first = lo;
    }
    for (int a = first + blockIdx.x; a < n_rows; a += gridDim.x) {
        const long long rb = max((long long)row_ptr[a], e0), re = min((long long)row_ptr[a + 1], e1);
        if (rb >= e1) break;
        if (a >= n_valid) {
            // no message gradient on this receiver: its edges hand over zeros
            for (long long e = rb; e < re; ++e) {
#pragma unroll
                for (int k = 0; k < IN; ++k) dxe[((e - dx0) * IN + k) * kC + c] = 0.0f;
                if (c == 0) qe[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
            continue;
        }
        float g_a[MID];
#pragma unroll
        for (int k = 0; k < MID; ++k) g_a[k] = __ldg(d_mid + ((long long)a * MID + k) * kC + c);
        for (long long batch = rb; batch < re; batch += kBatch) {
            const int nb = (int)min((long long)kBatch, re - batch);
            for (int k = 0; k < nb; ++k) {
                const long long e = batch + k;
                const int j = senders[e];
                float Y[16], w[P], wp[P], x_j[IN], dY[16], dxj[IN];
                {
                    const float4* yp = reinterpret_cast<const float4*>(edge_sh + 16 * e);
                    const float4 y0 = __ldg(yp), y1 = __ldg(yp + 1), y2 = __ldg(yp + 2), y3 = __ldg(yp + 3);
                    Y[0] = y0.x; Y[1] = y0.y; Y[2] = y0.z; Y[3] = y0.w; Y[4] = y1.x; Y[5] = y1.y; Y[6] = y1.z; Y[7] = y1.w;
                    Y[8] = y2.x; Y[9] = y2.y; Y[10] = y2.z; Y[11] = y2.w; Y[12] = y3.x; Y[13] = y3.y; Y[14] = y3.z; Y[15] = y3.w;
                }
                const float* wr = tp_w + (e - chunk_e0) * (long long)(P * kC) + c;
#pragma unroll
                for (int p = 0; p < P; ++p) {
                    w[p] = __ldg(wr + p * kC);
                    wp[p] = __ldg(wr + tangent_offset + p * kC);
                }
#pragma unroll
                for (int q = 0; q < IN; ++q) {
                    x_j[q] = __ldg(x + ((long long)j * IN + q) * kC + c);
                    dxj[q] = 0.0f;
                }
#pragma unroll
                for (int q = 0; q < 16; ++q) dY[q] = 0.0f;
                float dr = 0.0f;
                TpBackwardSel<LIN, false, true>::run(x_j, Y, w, wp, g_a, dY, dr, dxj);
#pragma unroll
                for (int q = 0; q < IN; ++q) dxe[((e - dx0) * IN + q) * kC + c] = dxj[q];
                // 16 + 1 sums over the channels: transpose-reduce inside the warp, the four warps meet in shared memory
                {
#pragma unroll
                    for (int half = 8, bit = 16; half >= 1; half >>= 1, bit >>= 1) {
                        const bool upper = (lane & bit) != 0;
#pragma unroll
                        for (int i = 0; i < half; ++i) {
                            const float keep = upper ? dY[i + half] : dY[i];
                            const float send = upper ? dY[i] : dY[i + half];
                            dY[i] = keep + __shfl_xor_sync(0xffffffffu, send, bit);
                        }
                    }
                    dY[0] += __shfl_xor_sync(0xffffffffu, dY[0], 1);
                }
                dr = warp_sum(dr);
                if ((lane & 1) == 0) red[k][warp][lane >> 1] = dY[0];
                if (lane == 0) red[k][warp][16] = dr;
            }
            __syncthreads();
            if (c < nb) {
                const long long e = batch + c;
                float g[16];
#pragma unroll
                for (int q = 0; q < 16; ++q) g[q] = red[c][0][q] + red[c][1][q] + red[c][2][q] + red[c][3][q];
                const float drt = red[c][0][16] + red[c][1][16] + red[c][2][16] + red[c][3][16];
                const float4 uv = __ldg(reinterpret_cast<const float4*>(edge_vec) + e);
                float q3[3];
                edge_vector_gradient(g, drt, uv.x, uv.y, uv.z, uv.w, q3);
                qe[e] = make_float4(q3[0], q3[1], q3[2], 0.0f);
            }
            __syncthreads();
        }
    }
}

// dE/dx_a = sum over the row of a of the hand-over of the mirror edges (rows at or beyond n_source hand over nothing; `end`:
// rows of dxe). With the comparison against `end` the compiler keeps the 36 loads of four edges of node l_max 2 in flight (47
// registers), without it it stops at 32 registers: force call of 1,728 atoms of the large model 1,443 against 1,458 us.
template <int IN>
__global__ void __launch_bounds__(kC)
k_gather_dx(int n_rows, int n_source, const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ senders,
            const int32_t* __restrict__ mirror, const float* __restrict__ dxe, float* __restrict__ d_x, long long end) {
    const int c = threadIdx.x;
    for (int a = blockIdx.x; a < n_rows; a += gridDim.x) {
        float acc[IN];
#pragma unroll
        for (int k = 0; k < IN; ++k) acc[k] = 0.0f;
        const long long rb = row_ptr[a], re = row_ptr[a + 1];
        // four edges at a time: their mirror indices first, then all the rows, so that the loads overlap
        for (long long e = rb; e < re; e += 4) {
            int m[4];
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const bool live = e + q < re;
                m[q] = live ? mirror[e + q] : -1;
                if (live && senders[e + q] >= n_source) m[q] = -1;
                if (m[q] >= end) m[q] = -1;
            }
            float v[4][IN];
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int k = 0; k < IN; ++k)
                    v[q][k] = m[q] >= 0 ? __ldg(dxe + ((long long)m[q] * IN + k) * kC + c) : 0.0f;
#pragma unroll
            for (int q = 0; q < 4; ++q)
#pragma unroll
                for (int k = 0; k < IN; ++k) acc[k] += v[q][k];
        }
#pragma unroll
        for (int k = 0; k < IN; ++k) d_x[((long long)a * IN + k) * kC + c] = acc[k];
    }
}

// The same for a buffer that holds the hand-over of the edges [first, end) only, added to what the chunks before gave
// (d_x starts from zero). Behind every chunk all atoms have to be asked, but the question is small: an edge's mirror lies
// in the chunk exactly when its sender is one of the chunk's receivers, and a row is sorted by sender, so one thread per
// atom finds the part of its row by two bisections and the warps then visit the atoms that have one -- an atom without
// reads some ten indices and neither reads nor writes d_x. The two receivers the chunk shares with its neighbours are
// decided by the mirror index. Order of the sums as in the kernel above.
// Latency of the two bisections and of a row's chain; a warp per row and 16 atoms a CTA keep that short on small lists
// (with a CTA per row: 7.4 and 21.5 ms for the second and third figure). Walking every row and rewriting d_x behind every
// chunk cost chunks times atoms. A whole force call in chunks of 2^19, 2^16 and 2^13 edges, before and after: 562 k edges
// 5.8 -> 5.7, 7.6 -> 6.7, 27.6 -> 18.3 ms; 3.54 M edges 40.3 -> 36, 96.5 -> 41 ms (2^19, 2^16); 28.3 M edges (884,736 atoms)
// 760 -> 307 ms (2^19).
constexpr int kGatherAtoms = 16;               // of a CTA

template <int IN>
__global__ void __launch_bounds__(128)
k_gather_dx_chunk(int n_rows, int n_source, const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ senders,
                  const int32_t* __restrict__ receivers, const int32_t* __restrict__ mirror, const float* __restrict__ dxe,
                  float* __restrict__ d_x, long long first, long long end) {
    constexpr int kAhead = IN > 4 ? 2 : 4;                     // edges whose rows are requested together
    __shared__ int part[2][kGatherAtoms];
    const int c = threadIdx.x, a0 = blockIdx.x * kGatherAtoms;
    end = min(end, (long long)row_ptr[n_source]);
    if (first >= end) return;
    if (c < 2 * kGatherAtoms) {
        // this atom's first edge whose sender is not below `bound`
        const int a = a0 + c % kGatherAtoms, upper = c / kGatherAtoms;
        int lo = 0;
        if (a < n_rows) {
            const int bound = upper ? receivers[end - 1] + 1 : receivers[first];
            lo = row_ptr[a];
            int hi = row_ptr[a + 1];
            while (lo < hi) {
                const int mid = (lo + hi) >> 1;
                if (senders[mid] < bound) lo = mid + 1; else hi = mid;
            }
        }
        part[upper][c % kGatherAtoms] = lo;
    }
    __syncthreads();
    // a warp per atom, four channels per lane
    const int lane = c & 31;
    for (int k = c >> 5; k < kGatherAtoms; k += 4) {
        const int rb = part[0][k], re = part[1][k];
        if (rb >= re) continue;
        float4* const row = reinterpret_cast<float4*>(d_x + (long long)(a0 + k) * IN * kC) + lane;
        float4 acc[IN];
#pragma unroll
        for (int q = 0; q < IN; ++q) acc[q] = row[q * (kC / 4)];
        for (int e = rb; e < re; e += kAhead) {
            int m[kAhead];
#pragma unroll
            for (int q = 0; q < kAhead; ++q) {
                m[q] = e + q < re ? mirror[e + q] : -1;
                if (m[q] < first || m[q] >= end) m[q] = -1;
            }
            float4 v[kAhead][IN];
#pragma unroll
            for (int q = 0; q < kAhead; ++q)
#pragma unroll
                for (int i = 0; i < IN; ++i)
                    v[q][i] = m[q] >= 0 ? __ldg(reinterpret_cast<const float4*>(dxe + ((m[q] - first) * IN + i) * kC) + lane)
                                        : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
            for (int q = 0; q < kAhead; ++q)
#pragma unroll
                for (int i = 0; i < IN; ++i) {
                    acc[i].x += v[q][i].x; acc[i].y += v[q][i].y; acc[i].z += v[q][i].z; acc[i].w += v[q][i].w;
                }
        }
#pragma unroll
        for (int q = 0; q < IN; ++q) row[q * (kC / 4)] = acc[q];
    }
}

// First interaction (reassociated form), per edge: the receiver's gradient block [16][Z][64] in shared memory,
// dE/dY[lm] = sum_k dS[lm, z_j, k] hidden[k], dE/dr = sum_k hidden'[k] sum_lm dS[lm, z_j, k] Y[lm]; the edge-vector
// gradient is added to qe (rows below n_add, which the later interaction wrote) or stored. A thread takes an edge and
// four harmonics: the sums over the 64 radial features run inside the thread -- the features of 16 edges are staged in
// shared memory -- and only the four threads of an edge meet at the end, by shuffles inside a group of four lanes. (A
// thread per (feature, eight harmonics) spent 137 instructions per warp and edge on 16 FMAs per thread: channel
// reductions by shuffle and two barriers per eight edges; 72 -> 45 us.)
// The features of 16 edges arrive by asynchronous copies a pass ahead, and features and gradient block are read four
// values at a time: with single values the six shared-memory reads per nine FMAs bounded the kernel (42 -> 35 us at 62 k
// edges, 217 -> 197 us at 615 k, 431 -> 330 us at 748 k edges and five species).
constexpr int kFaPass = 16;                       // edges per pass
constexpr int kFaThreads = 4 * kFaPass;
constexpr int kFaLd = kRadial + 4;                // row stride: 16-byte rows, neighbouring rows start four banks apart

// Floats from one group of four harmonics to the next in the gradient block: 8 mod 32, so that the four groups and two
// neighbouring species are read from different banks.
__host__ __device__ constexpr int fa_group(int n_species) {
    const int rows = 4 * n_species * kFaLd;
    return rows + (8 - rows % 32 + 32) % 32;
}

__device__ __forceinline__ void copy_row_part(float* dst, const float* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" :: "r"(tc::smem_u32(dst)), "l"(src) : "memory");
}

__global__ void __launch_bounds__(kFaThreads)
k_first_adjoint_rows(int n_rows, int n_valid, int n_add, int n_species, const int32_t* __restrict__ row_ptr,
                     const int32_t* __restrict__ senders, const int32_t* __restrict__ species,
                     const float* __restrict__ edge_sh, const float* __restrict__ edge_vec,
                     const float* __restrict__ hidden, const float* __restrict__ hidden_tangent,
                     const float* __restrict__ d_s, float4* __restrict__ qe, const float* __restrict__ parts, long long part_stride) {
    extern __shared__ __align__(16) float staged[];       // [2 buffers][values, tangents][kFaPass][kFaLd]
    float* const own = staged + 4 * kFaPass * kFaLd;      // [4 groups][4][n_species][kFaLd]
    const int c = threadIdx.x, slot = c >> 2, grp = c & 3, lane = c & 31;
    const int row_floats = kNSH * n_species * kRadial;
    const int lm_stride = n_species * kFaLd, group = fa_group(n_species);
    auto stage = [&](long long first, long long re, int buf) {
        const int nb = (int)min((long long)kFaPass, re - first);
        float* const to = staged + buf * 2 * kFaPass * kFaLd;
        for (int q = c; q < nb * (kRadial / 4); q += kFaThreads) {
            const int el = q >> 4, k = 4 * (q & 15);
            copy_row_part(to + el * kFaLd + k, hidden + (first + el) * kRadial + k);
            copy_row_part(to + (kFaPass + el) * kFaLd + k, hidden_tangent + (first + el) * kRadial + k);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    for (int a = blockIdx.x; a < n_rows; a += gridDim.x) {
        const long long rb = row_ptr[a], re = row_ptr[a + 1];
        if (a >= n_valid) {
            if (a >= n_add)
                for (long long e = rb + c; e < re; e += kFaThreads) qe[e] = make_float4(0.f, 0.f, 0.f, 0.f);
            continue;
        }
        if (rb >= re) continue;
        // the previous row's last barrier freed its block and both buffers
        for (int q = c; q < row_floats / 4; q += kFaThreads)
            copy_row_part(own + (q >> 4) * kFaLd + ((q >> 4) / (4 * n_species)) * (group - 4 * lm_stride) + 4 * (q & 15),
                          d_s + (long long)a * row_floats + 4 * q);
        stage(rb, re, 0);
        int z_next = rb + slot < re ? species[senders[rb + slot]] : 0;
        int buf = 0;
        for (long long batch = rb; batch < re; batch += kFaPass, buf ^= 1) {
            const int nb = (int)min((long long)kFaPass, re - batch);
            const int zj = z_next;
            if (batch + kFaPass < re) {
                stage(batch + kFaPass, re, buf ^ 1);
                const long long e = batch + kFaPass + slot;
                z_next = e < re ? species[senders[e]] : 0;
                asm volatile("cp.async.wait_group 1;" ::: "memory");
            } else {
                asm volatile("cp.async.wait_group 0;" ::: "memory");
            }
            __syncthreads();
            const bool live = slot < nb;
            const long long e = batch + (live ? slot : 0);
            float g[4] = {0.f, 0.f, 0.f, 0.f}, dr = 0.0f;
            if (live) {
                const float4 y = __ldg(reinterpret_cast<const float4*>(edge_sh + 16 * e) + grp);
                const float4* hs = reinterpret_cast<const float4*>(staged + (buf * 2 * kFaPass + slot) * kFaLd);
                const float4* hps = hs + kFaPass * kFaLd / 4;
                const float4* ds = reinterpret_cast<const float4*>(own + grp * group + zj * kFaLd);     // harmonics 4 grp ..
                const int next = lm_stride / 4;
                auto term = [&](float h, float hp, float d0, float d1, float d2, float d3) {
                    g[0] = fmaf(d0, h, g[0]); g[1] = fmaf(d1, h, g[1]); g[2] = fmaf(d2, h, g[2]); g[3] = fmaf(d3, h, g[3]);
                    dr = fmaf(fmaf(d0, y.x, fmaf(d1, y.y, fmaf(d2, y.z, d3 * y.w))), hp, dr);
                };
#pragma unroll 4
                for (int k = 0; k < kRadial / 4; ++k) {
                    const float4 h = hs[k], hp = hps[k], d0 = ds[k], d1 = ds[next + k], d2 = ds[2 * next + k], d3 = ds[3 * next + k];
                    term(h.x, hp.x, d0.x, d1.x, d2.x, d3.x);
                    term(h.y, hp.y, d0.y, d1.y, d2.y, d3.y);
                    term(h.z, hp.z, d0.z, d1.z, d2.z, d3.z);
                    term(h.w, hp.w, d0.w, d1.w, d2.w, d3.w);
                }
            }
            if (live && parts && a < n_add) {
#pragma unroll
                for (int half = 0; half < 2; ++half) {
                    const float* const from = parts + (half * part_stride + e) * 20;
                    const float4 more = __ldg(reinterpret_cast<const float4*>(from) + grp);
                    g[0] += more.x; g[1] += more.y; g[2] += more.z; g[3] += more.w;
                    if (grp == 0) dr += __ldg(from + 16);
                }
            }
            // the four threads of an edge exchange their harmonics' gradients and add up the radial one
            float all[16];
            const int base = lane & ~3;
#pragma unroll
            for (int src = 0; src < 4; ++src)
#pragma unroll
                for (int i = 0; i < 4; ++i) all[4 * src + i] = __shfl_sync(0xffffffffu, g[i], base + src);
            dr += __shfl_xor_sync(0xffffffffu, dr, 1);
            dr += __shfl_xor_sync(0xffffffffu, dr, 2);
            if (live && grp == 0) {
                const float4 uv = __ldg(reinterpret_cast<const float4*>(edge_vec) + e);
                float q3[3];
                edge_vector_gradient(all, dr, uv.x, uv.y, uv.z, uv.w, q3);
                float4 out = make_float4(q3[0], q3[1], q3[2], 0.0f);
                if (a < n_add && !parts) {
                    const float4 old = qe[e];
                    out.x += old.x; out.y += old.y; out.z += old.z;
                }
                qe[e] = out;
            }
            __syncthreads();                              // the pass is done with its buffer (and, at the end, with the block)
        }
    }
}

// F_a = -(sum_row qe[e] - qe[mirror e]), virial_a = sum_row v_e (x) qe[e]; one warp per atom, lanes over its edges,
// folded with a fixed butterfly. RESTRICT: only the edges into atoms below n_valid carry a gradient -- an atom at or
// beyond it (a halo atom) has no row terms and no virial, and a mirror edge counts only if its receiver (this edge's
// sender) is below n_valid; qe and edge_vec are never read elsewhere.
template <bool RESTRICT>
__global__ void __launch_bounds__(256)
k_force_gather(int n_atoms, int n_valid, const int32_t* __restrict__ row_ptr, const int32_t* __restrict__ senders,
               const int32_t* __restrict__ mirror, const float4* __restrict__ qe, const float* __restrict__ edge_vec,
               float* __restrict__ force_acc, float* __restrict__ atom_virial) {
    const int a = blockIdx.x * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (a >= n_atoms) return;
    float f[3] = {0.f, 0.f, 0.f}, vir[6] = {0.f, 0.f, 0.f, 0.f, 0.f, 0.f};
    const bool own = !RESTRICT || a < n_valid;
    for (long long e = row_ptr[a] + lane; e < row_ptr[a + 1]; e += 32) {
        const float4 q = own ? qe[e] : make_float4(0.f, 0.f, 0.f, 0.f);
        int m = mirror[e];
        if (RESTRICT && senders[e] >= n_valid) m = -1;
        const float4 qm = m >= 0 ? qe[m] : make_float4(0.f, 0.f, 0.f, 0.f);
        f[0] += q.x - qm.x; f[1] += q.y - qm.y; f[2] += q.z - qm.z;
        if (own) {
            const float4 uv = __ldg(reinterpret_cast<const float4*>(edge_vec) + e);
            const float vx = uv.x * uv.w, vy = uv.y * uv.w, vz = uv.z * uv.w;
            vir[0] += vx * q.x; vir[1] += vy * q.y; vir[2] += vz * q.z;
            vir[3] += 0.5f * (vy * q.z + vz * q.y);
            vir[4] += 0.5f * (vx * q.z + vz * q.x);
            vir[5] += 0.5f * (vx * q.y + vy * q.x);
        }
    }
#pragma unroll
    for (int q = 0; q < 3; ++q) f[q] = warp_sum(f[q]);
#pragma unroll
    for (int q = 0; q < 6; ++q) vir[q] = warp_sum(vir[q]);
    if (lane == 0) {
#pragma unroll
        for (int q = 0; q < 3; ++q) force_acc[3 * (long long)a + q] = f[q];
#pragma unroll
        for (int q = 0; q < 6; ++q) atom_virial[6 * (long long)a + q] = vir[q];
    }
}

template <int IN>
int gather_launch(const EdgeAdjointArgs& t, int rows, bool chunk, cudaStream_t stream) {
    if (chunk) {
        if (t.chunk_e0 == 0) FMB_CUDA_CHECK(cudaMemsetAsync(t.d_x, 0, (size_t)rows * IN * kC * sizeof(float), stream));
        k_gather_dx_chunk<IN><<<ceil_div(rows, kGatherAtoms), 128, 0, stream>>>(
            rows, t.n_rows, t.row_ptr, t.senders, t.receivers, t.mirror, t.dxe, t.d_x, t.chunk_e0, t.chunk_e0 + t.chunk_edges);
    } else {
        k_gather_dx<IN><<<rows < 1184 ? rows : 1184, kC, 0, stream>>>(rows, t.n_rows, t.row_ptr, t.senders, t.mirror, t.dxe,
                                                                      t.d_x, t.dx_rows);
    }
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

int grid_for(const void* kernel, int rows, int threads, size_t smem) {
    int per_sm = 0, sms = 148, dev = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kernel, threads, smem) != cudaSuccess || per_sm < 1) per_sm = 1;
    if (cudaGetDevice(&dev) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    const int cap = per_sm * sms * 4;
    return rows < cap ? rows : cap;
}

}  // namespace

int mirror_map(const fmb_nl_t* nl, int32_t* mirror, uint32_t* status, const long long* listed_below, int32_t* slot,
               int32_t* list, long long* list_count, int list_capacity, cudaStream_t stream) {
    const int blocks = ceil_div(nl->capacity, 256);
    if (slot) FMB_CUDA_CHECK(cudaMemsetAsync(list_count, 0, sizeof(long long), stream));
    k_mirror<<<blocks < 1184 ? blocks : 1184, 256, 0, stream>>>((const long long*)nl->count, nl->capacity, nl->edge_index,
                                                               nl->unit_shifts, nl->edge_row_ptr, mirror, status,
                                                               listed_below, slot, list, (unsigned long long*)list_count,
                                                               list_capacity);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

int tp_adjoint_edges(const EdgeAdjointArgs& t, cudaStream_t stream) {
    if (t.n_rows <= 0) return FMB_OK;
    if (t.n_valid >= t.n_rows) return tp_adjoint_coupled_launch(t, stream);
    if (t.lin == 0) {
        static const int grid_cap = grid_for((const void*)k_tp_adjoint_edges<0, 2>, 1 << 30, kC, 0);
        k_tp_adjoint_edges<0, 2><<<t.n_rows < grid_cap ? t.n_rows : grid_cap, kC, 0, stream>>>(
            t.n_atoms, t.n_rows, t.n_valid, t.chunk_e0, t.chunk_edges, t.count, t.row_ptr, t.senders, t.x, t.edge_sh, t.edge_vec,
            t.tp_w, t.tangent_offset, t.d_mid, t.dxe, reinterpret_cast<float4*>(t.qe), t.dx_e0);
    } else if (t.lin == 1) {
        // four CTAs per SM (127 registers): measured best on the 1,944-atom cell among 2 .. 6
        static const int grid_cap = grid_for((const void*)k_tp_adjoint_edges<1, 4>, 1 << 30, kC, 0);
        k_tp_adjoint_edges<1, 4><<<t.n_rows < grid_cap ? t.n_rows : grid_cap, kC, 0, stream>>>(
            t.n_atoms, t.n_rows, t.n_valid, t.chunk_e0, t.chunk_edges, t.count, t.row_ptr, t.senders, t.x, t.edge_sh,
            t.edge_vec, t.tp_w, t.tangent_offset, t.d_mid, t.dxe, reinterpret_cast<float4*>(t.qe), t.dx_e0);
    } else if (t.lin == 2) {
        static const int grid_cap = grid_for((const void*)k_tp_adjoint_edges<2, 2>, 1 << 30, kC, 0);
        k_tp_adjoint_edges<2, 2><<<t.n_rows < grid_cap ? t.n_rows : grid_cap, kC, 0, stream>>>(
            t.n_atoms, t.n_rows, t.n_valid, t.chunk_e0, t.chunk_edges, t.count, t.row_ptr, t.senders, t.x, t.edge_sh, t.edge_vec,
            t.tp_w, t.tangent_offset, t.d_mid, t.dxe, reinterpret_cast<float4*>(t.qe), t.dx_e0);
    } else {
        return FMB_ERR_UNSUPPORTED;
    }
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

int gather_sender_gradient(const EdgeAdjointArgs& t, bool chunk, cudaStream_t stream) {
    const int rows = t.n_gather > 0 ? t.n_gather : t.n_rows;     // atoms that collect; the edges of [0, n_rows) hand over
    if (rows <= 0) return FMB_OK;
    if (t.lin == 0) return gather_launch<1>(t, rows, chunk, stream);
    if (t.lin == 1) return gather_launch<4>(t, rows, chunk, stream);
    if (t.lin == 2) return gather_launch<9>(t, rows, chunk, stream);
    return FMB_ERR_UNSUPPORTED;
}

int first_adjoint_edges(const FirstArgs& f, int n_add, float* qe, const float* parts, long long part_stride, cudaStream_t stream) {
    if (f.n_rows <= 0) return FMB_OK;
    const size_t smem = (size_t)(4 * fa_group(f.n_species) + 4 * kFaPass * kFaLd) * sizeof(float);
    FMB_CUDA_CHECK(opt_in_shared_memory((const void*)k_first_adjoint_rows,
                                        (4 * fa_group(FMB_MAX_SPECIES) + 4 * kFaPass * kFaLd) * (int)sizeof(float)));
    const int grid_cap = grid_for((const void*)k_first_adjoint_rows, 1 << 30, kFaThreads, smem);
    k_first_adjoint_rows<<<f.n_rows < grid_cap ? f.n_rows : grid_cap, kFaThreads, smem, stream>>>(
        f.n_rows, f.n_valid, n_add, f.n_species, f.row_ptr, f.senders, f.species, f.edge_sh, f.edge_vec, f.hidden,
        f.hidden_tangent, f.d_s, reinterpret_cast<float4*>(qe), parts, part_stride);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

int force_gather(int n_atoms, int n_valid, const int32_t* row_ptr, const int32_t* senders, const int32_t* mirror,
                 const float* qe, const float* edge_vec, float* force_acc, float* atom_virial, cudaStream_t stream) {
    if (n_atoms <= 0) return FMB_OK;
    if (n_valid < n_atoms)
        k_force_gather<true><<<ceil_div(n_atoms, 8), 256, 0, stream>>>(n_atoms, n_valid, row_ptr, senders, mirror,
                                                                       reinterpret_cast<const float4*>(qe), edge_vec,
                                                                       force_acc, atom_virial);
    else
        k_force_gather<false><<<ceil_div(n_atoms, 8), 256, 0, stream>>>(n_atoms, n_valid, row_ptr, senders, mirror,
                                                                        reinterpret_cast<const float4*>(qe), edge_vec,
                                                                        force_acc, atom_virial);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

}  // namespace fmb
