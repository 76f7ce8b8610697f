// Per-atom stages: readouts with their gradient, the float64 energy / virial reductions.
//
// Reference: energy contract fastmace/model/energy.py:92-99 (per-atom terms in model precision, reduced in float64, E0
// in float64).

#include "stages.cuh"
#include "fold.cuh"

namespace fmb {

namespace {

// h[a][k][c] = table[species[a]][k][c]  (layer 0's species-only skip connection)
__global__ void k_fill_from_species(int n_atoms, int row, const int32_t* __restrict__ species,
                                    const float* __restrict__ table, float* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)n_atoms * row) return;
    const int a = (int)(i / row), k = (int)(i % row);
    out[i] = table[(long long)species[a] * row + k];
}

// A warp per atom, four channels per lane, the weights of both readouts in registers for all the atoms it visits. Non-last
// layers: e += h[a][0][:] . w, gradient w. Last layer: 128 -> 16 -> SiLU -> 1 with its gradient. The energy scale is folded
// in here. Bound by the rows it writes (the gradient of the first layer's features, zeros but for the scalars), on small
// systems by its chain. With the weights read again for every atom (64 strided loads, twice) and every sum a butterfly of its
// own 62 -> 13 us for 10,368 atoms of the middle model, 14.5 -> 8.5 for 1,944.
constexpr int kReadoutWarps = 4;
__global__ void __launch_bounds__(32 * kReadoutWarps)
k_readout(int n_atoms, int n_energy, int dim_first, int dim_last, float scale, float shift, float silu_norm,
          const float* __restrict__ h_first, const float* __restrict__ h_last, const float* __restrict__ w_first,
          const float* __restrict__ w_last0, const float* __restrict__ w_last1, float* __restrict__ node_energy,
          float* __restrict__ d_h_first, float* __restrict__ d_h_last) {
    const int lane = threadIdx.x & 31, warps = gridDim.x * kReadoutWarps;
    const bool wide = ((reinterpret_cast<uintptr_t>(w_first) | reinterpret_cast<uintptr_t>(w_last0)) & 15) == 0;
    auto weights = [wide](const float* from) {
        return wide ? __ldg(reinterpret_cast<const float4*>(from)) : make_float4(__ldg(from), __ldg(from + 1), __ldg(from + 2), __ldg(from + 3));
    };
    const float4 wf = weights(w_first + 4 * lane);
    float w[4][16];                            // of channels 4 lane .. 4 lane + 3
#pragma unroll
    for (int c = 0; c < 4; ++c)
#pragma unroll
        for (int j = 0; j < 16; j += 4) {
            const float4 v = weights(w_last0 + (4 * lane + c) * 16 + j);
            w[c][j] = v.x; w[c][j + 1] = v.y; w[c][j + 2] = v.z; w[c][j + 3] = v.w;
        }
    const float w1 = __ldg(w_last1 + (lane >> 1));         // `fold` leaves sum j of 16 in the lanes 2 j and 2 j + 1
    for (int a = blockIdx.x * kReadoutWarps + (threadIdx.x >> 5); a < n_atoms; a += warps) {
        float4* const df = reinterpret_cast<float4*>(d_h_first + (long long)a * dim_first * kC) + lane;
        const float4 zero = make_float4(0.f, 0.f, 0.f, 0.f);
        for (int k = 1; k < dim_first; ++k) df[k * (kC / 4)] = zero;
        if (a >= n_energy) {
            // an atom whose energy belongs to another domain: it contributes no energy and seeds no gradient
            df[0] = zero;
            if (lane == 0) node_energy[a] = 0.0f;
            continue;
        }
        // first readout (linear) and the gradient it leaves on h_first's scalars; other components start at zero
        const float4 hf = __ldg(reinterpret_cast<const float4*>(h_first + (long long)a * dim_first * kC) + lane);
        const float4 hl = __ldg(reinterpret_cast<const float4*>(h_last + (long long)a * dim_last * kC) + lane);
        float e = fmaf(hf.x, wf.x, fmaf(hf.y, wf.y, fmaf(hf.z, wf.z, hf.w * wf.w)));
        df[0] = make_float4(scale * wf.x, scale * wf.y, scale * wf.z, scale * wf.w);
        // last readout
        float z[16];
#pragma unroll
        for (int j = 0; j < 16; ++j) z[j] = fmaf(hl.x, w[0][j], fmaf(hl.y, w[1][j], fmaf(hl.z, w[2][j], hl.w * w[3][j])));
        fold<16, 16>(z, lane);
        const float zz = z[0], sig = 1.0f / (1.0f + expf(-zz));
        if ((lane & 1) == 0) e += silu_norm * zz * sig * w1;          // two lanes hold every sum
        const float dz = scale * w1 * silu_norm * sig * (1.0f + zz * (1.0f - sig));
        e = warp_sum(e);
        if (lane == 0) node_energy[a] = scale * e + shift;
        float g[4] = {0.f, 0.f, 0.f, 0.f};
#pragma unroll
        for (int j = 0; j < 16; ++j) {
            const float d = __shfl_sync(0xffffffffu, dz, 2 * j);
#pragma unroll
            for (int c = 0; c < 4; ++c) g[c] = fmaf(w[c][j], d, g[c]);
        }
        reinterpret_cast<float4*>(d_h_last + (long long)a * dim_last * kC)[lane] = make_float4(g[0], g[1], g[2], g[3]);
    }
}

constexpr int kReduceBlocks = 256;

struct E0Table {
    double v[FMB_MAX_SPECIES];
};

// partial[b][0] = sum of node energies (+E0) of block b's atoms, partial[b][1..6] = virial components; float64.
__global__ void __launch_bounds__(256)
k_reduce_partial(int n_atoms, int n_energy, const float* __restrict__ node_energy, const int32_t* __restrict__ species,
                 E0Table e0, const float* __restrict__ atom_virial,
                 double* __restrict__ partial, const float* __restrict__ force_acc, float* __restrict__ forces) {
    __shared__ double sh[8][7];
    // the forces are minus the accumulated gradient (independent of the sums below; it saves a launch)
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < 3 * n_atoms; i += gridDim.x * blockDim.x) forces[i] = -force_acc[i];
    double acc[7] = {0, 0, 0, 0, 0, 0, 0};
    const int per_block = (n_atoms + gridDim.x - 1) / gridDim.x;
    const int begin = blockIdx.x * per_block, end = min(n_atoms, begin + per_block);
    for (int a = begin + threadIdx.x; a < end; a += blockDim.x) {
        if (a < n_energy) acc[0] += (double)node_energy[a] + e0.v[species[a]];
        if (atom_virial) {
#pragma unroll
            for (int q = 0; q < 6; ++q) acc[1 + q] += (double)atom_virial[6 * a + q];
        }
    }
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
#pragma unroll
    for (int q = 0; q < 7; ++q) {
        const double v = warp_sum(acc[q]);
        if (lane == 0) sh[warp][q] = v;
    }
    __syncthreads();
    if (threadIdx.x < 7) {
        double v = 0.0;
        for (int w = 0; w < 8; ++w) v += sh[w][threadIdx.x];
        partial[blockIdx.x * 8 + threadIdx.x] = v;
    }
}

// one warp per quantity (energy, six virial components): lane l adds blocks l, l + 32, ... in order, then a butterfly
// in fixed order -- the same sum every run
__global__ void __launch_bounds__(7 * 32)
k_reduce_final(int blocks, const double* __restrict__ partial, double inv_volume, int compute_stress,
               double* __restrict__ energy, float* __restrict__ stress, uint32_t* __restrict__ status) {
    const int q = threadIdx.x >> 5, lane = threadIdx.x & 31;
    double v = 0.0;
    for (int b = lane; b < blocks; b += 32) v += partial[b * 8 + q];
    v = warp_sum(v);
    if (lane != 0) return;
    if (q == 0) {
        *energy = v;
        if (!(v == v) || v > 1e300 || v < -1e300) atomicOr(status, FMB_STATUS_NONFINITE);
    } else if (compute_stress) {
        // order xx, yy, zz, yz, xz, xy
        const double s = v * inv_volume;
        const int idx[6][2] = {{0, 0}, {1, 1}, {2, 2}, {1, 2}, {0, 2}, {0, 1}};
        const int i = idx[q - 1][0], j = idx[q - 1][1];
        stress[3 * i + j] = (float)s;
        stress[3 * j + i] = (float)s;
    }
}

__global__ void k_commit(int n3, const float* __restrict__ forces, const double* __restrict__ energy,
                         const float* __restrict__ stress, double* __restrict__ f64, double* __restrict__ e64,
                         double* __restrict__ s64) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n3) f64[i] = (double)forces[i];
    if (i == 0) *e64 = *energy;
    if (s64 && i < 9) s64[i] = (double)stress[i];
}

}  // namespace

int fill_from_species(int n_atoms, int row, const int32_t* species, const float* table, float* out, cudaStream_t stream) {
    const long long total = (long long)n_atoms * row;
    k_fill_from_species<<<ceil_div(total, 256), 256, 0, stream>>>(n_atoms, row, species, table, out);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

int readout(const fmb_model_t* m, int n_atoms, int n_energy, const float* h_first, const float* h_last,
            float* node_energy, float* d_h_first, float* d_h_last, cudaStream_t stream) {
    const int dim_first = (m->layer[0].l_out_max + 1) * (m->layer[0].l_out_max + 1);
    const int dim_last = 1;
    const float* w_last = m->layer[m->n_layers - 1].w_readout;
    static const int cap = [] {                // four CTAs per SM
        int device = 0, sms = 148;
        if (cudaGetDevice(&device) == cudaSuccess) cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, device);
        return 4 * sms;
    }();
    const int blocks = ceil_div(n_atoms, kReadoutWarps);
    k_readout<<<blocks < cap ? blocks : cap, 32 * kReadoutWarps, 0, stream>>>(
        n_atoms, n_energy, dim_first, dim_last, m->scale, m->shift, m->silu_norm, h_first, h_last, m->layer[0].w_readout, w_last,
        w_last + kC * 16, node_energy, d_h_first, d_h_last);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

int reduce_outputs(const fmb_model_t* m, const fmb_work_t* w, int n_energy, double volume, cudaStream_t stream) {
    E0Table e0;
    for (int k = 0; k < FMB_MAX_SPECIES; ++k) e0.v[k] = m->e0[k];
    k_reduce_partial<<<kReduceBlocks, 256, 0, stream>>>(w->n_atoms, n_energy, w->node_energy, w->species, e0,
                                                        w->compute_stress ? w->atom_virial : nullptr, w->partial,
                                                        w->force_acc, w->forces);
    FMB_LAUNCH_CHECK();
    k_reduce_final<<<1, 7 * 32, 0, stream>>>(kReduceBlocks, w->partial, 1.0 / volume, w->compute_stress, w->energy, w->stress,
                                         w->status);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

int commit_forces(const fmb_work_t* w, double* f64, double* e64, double* s64, cudaStream_t stream) {
    k_commit<<<ceil_div(3LL * w->n_atoms, 256), 256, 0, stream>>>(3 * w->n_atoms, w->forces, w->energy, w->stress, f64,
                                                                  e64, s64);
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

}  // namespace fmb
