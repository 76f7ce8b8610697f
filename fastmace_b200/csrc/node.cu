// Per-atom stages: symmetric contraction (correlation 3) as a species-dependent polynomial in the 16 message
// components, readouts with their gradient, the float64 energy / virial reductions.
//
// Reference: EquivariantProductBasisBlock / SymmetricContraction of mace-torch, in the polynomial form the reference's
// generated kernels evaluate (fastmace/kernels/cuda/sc_generated.py:1-20: one block per atom, one thread per
// channel, y_C = sum_a w_a sum coef * monomial); energy contract fastmace/model/energy.py:92-99 (per-atom terms in
// model precision, reduced in float64, E0 in float64).

#include "stages.cuh"
#include "generated/symcon_generated.cuh"

namespace fmb {

namespace {

// One thread per (atom, channel); the polynomial is generated straight-line code (generated/symcon_generated.cuh):
// 16 inputs and the outputs live in registers, each coefficient is one coalesced load from the [species][term][C] table.
template <int LOUT>
__global__ void __launch_bounds__(kC)
k_symcon_forward(int n_atoms, int n_terms, const float* __restrict__ coef, const int32_t* __restrict__ species,
                 const float* __restrict__ msg, float* __restrict__ basis) {
    constexpr int OUT = SymconShape<LOUT>::kOut;
    const int a = blockIdx.x, c = threadIdx.x;
    if (a >= n_atoms) return;
    float x[kNSH], y[OUT];
#pragma unroll
    for (int k = 0; k < kNSH; ++k) x[k] = msg[((long long)a * kNSH + k) * kC + c];
#pragma unroll
    for (int k = 0; k < OUT; ++k) y[k] = 0.0f;
    symcon_forward_body<LOUT>(x, coef + (long long)species[a] * n_terms * kC + c, y);
#pragma unroll
    for (int k = 0; k < OUT; ++k) basis[((long long)a * OUT + k) * kC + c] = y[k];
}

template <int LOUT>
__global__ void __launch_bounds__(kC)
k_symcon_backward(int n_atoms, int n_terms, const float* __restrict__ coef, const int32_t* __restrict__ species,
                  const float* __restrict__ msg, const float* __restrict__ d_basis, float* __restrict__ d_msg) {
    constexpr int OUT = SymconShape<LOUT>::kOut;
    const int a = blockIdx.x, c = threadIdx.x;
    if (a >= n_atoms) return;
    float x[kNSH], dx[kNSH], g[OUT];
#pragma unroll
    for (int k = 0; k < kNSH; ++k) {
        x[k] = msg[((long long)a * kNSH + k) * kC + c];
        dx[k] = 0.0f;
    }
#pragma unroll
    for (int k = 0; k < OUT; ++k) g[k] = d_basis[((long long)a * OUT + k) * kC + c];
    symcon_backward_body<LOUT>(x, coef + (long long)species[a] * n_terms * kC + c, g, dx);
#pragma unroll
    for (int k = 0; k < kNSH; ++k) d_msg[((long long)a * kNSH + k) * kC + c] = dx[k];
}

// The same for the four atoms of a group (one species; -1 = empty slot; atoms at or beyond n_rows are skipped): a
// coefficient is loaded once and used for two pairs of atoms on the packed FP32 pipe. A CTA takes CH of the 128 channels;
// PARTS sets of CH threads share them, each with a run of the monomials, and their sums meet in shared memory.
//
// Bound: the coefficient table that a group streams from L2 (48, 210 or 454 KB for outputs up to l = 0, 1, 2), and with few
// groups the chain of a thread's terms. Two atoms at a time on scalar instructions, as before: 1,944 atoms 41 -> 31 us
// forward (both layers), 10,368 atoms 117 -> 83 and 170 -> 148 us, 13,824 atoms of the large model 445 -> 183 and
// 364 -> 294 us.
__device__ __forceinline__ int group_member(const int32_t* __restrict__ groups, int group, int slot, int n_rows) {
    const int atom = groups[4 * group + slot];
    return atom < n_rows ? atom : -1;
}

template <int K>
__device__ __forceinline__ void load_pairs(const float* __restrict__ rows, const int (&atom)[4], int c, float2 (&v)[2][K]) {
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int k = 0; k < K; ++k) {
            v[r][k].x = atom[2 * r] >= 0 ? rows[((long long)atom[2 * r] * K + k) * kC + c] : 0.0f;
            v[r][k].y = atom[2 * r + 1] >= 0 ? rows[((long long)atom[2 * r + 1] * K + k) * kC + c] : 0.0f;
        }
}

// adds the parts' values into those of part 0 (pairwise: half of the parts hand over at a time)
template <int K, int PARTS, int CH>
__device__ __forceinline__ void add_parts(float2 (&v)[2][K], int part, int c, float2* shared) {
#pragma unroll
    for (int half = PARTS / 2; half >= 1; half >>= 1) {
        float2* const slot = shared + (part & (half - 1)) * 2 * K * CH + c;
        if (part >= half && part < 2 * half) {
#pragma unroll
            for (int q = 0; q < 2 * K; ++q) slot[q * CH] = v[q / K][q % K];
        }
        __syncthreads();
        if (part < half) {
#pragma unroll
            for (int q = 0; q < 2 * K; ++q) {
                const float2 o = slot[q * CH];
                v[q / K][q % K].x += o.x;
                v[q / K][q % K].y += o.y;
            }
        }
        if (half > 1) __syncthreads();
    }
}

template <int K>
__device__ __forceinline__ void store_pairs(float* __restrict__ rows, const int (&atom)[4], int c, const float2 (&v)[2][K]) {
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int k = 0; k < K; ++k) {
            if (atom[2 * r] >= 0) rows[((long long)atom[2 * r] * K + k) * kC + c] = v[r][k].x;
            if (atom[2 * r + 1] >= 0) rows[((long long)atom[2 * r + 1] * K + k) * kC + c] = v[r][k].y;
        }
}

template <int LOUT, int PARTS, int CH, int MINB>
__global__ void __launch_bounds__(CH * PARTS, MINB)
k_symcon_forward_group(int n_rows, const float* __restrict__ coef, const int32_t* __restrict__ species,
                       const int32_t* __restrict__ groups, const float* __restrict__ msg, float* __restrict__ basis) {
    constexpr int OUT = SymconShape<LOUT>::kOut;
    extern __shared__ float2 shared[];
    const int group = blockIdx.x / (kC / CH), t = threadIdx.x % CH, part = threadIdx.x / CH;
    const int c = t + CH * (blockIdx.x % (kC / CH));
    const int atom[4] = {group_member(groups, group, 0, n_rows), group_member(groups, group, 1, n_rows),
                         group_member(groups, group, 2, n_rows), group_member(groups, group, 3, n_rows)};
    const int lead = max(max(atom[0], atom[1]), max(atom[2], atom[3]));
    if (lead < 0) return;
    float2 x[2][kNSH], y[2][OUT];
    load_pairs(msg, atom, c, x);
#pragma unroll
    for (int q = 0; q < 2 * OUT; ++q) y[q / OUT][q % OUT] = make_float2(0.0f, 0.0f);
    symcon_forward_group<LOUT, PARTS>(part, x, coef + (long long)species[lead] * SymconShape<LOUT>::kTerms * kC + c, y);
    add_parts<OUT, PARTS, CH>(y, part, t, shared);
    if (part == 0) store_pairs(basis, atom, c, y);
}

template <int LOUT, int PARTS, int CH, int MINB>
__global__ void __launch_bounds__(CH * PARTS, MINB)
k_symcon_backward_group(int n_rows, const float* __restrict__ coef, const int32_t* __restrict__ species,
                        const int32_t* __restrict__ groups, const float* __restrict__ msg, const float* __restrict__ d_basis,
                        float* __restrict__ d_msg) {
    constexpr int OUT = SymconShape<LOUT>::kOut;
    extern __shared__ float2 shared[];
    const int group = blockIdx.x / (kC / CH), t = threadIdx.x % CH, part = threadIdx.x / CH;
    const int c = t + CH * (blockIdx.x % (kC / CH));
    const int atom[4] = {group_member(groups, group, 0, n_rows), group_member(groups, group, 1, n_rows),
                         group_member(groups, group, 2, n_rows), group_member(groups, group, 3, n_rows)};
    const int lead = max(max(atom[0], atom[1]), max(atom[2], atom[3]));
    if (lead < 0) return;
    float2 x[2][kNSH], dx[2][kNSH], g[2][OUT];
    load_pairs(msg, atom, c, x);
    load_pairs(d_basis, atom, c, g);
#pragma unroll
    for (int q = 0; q < 2 * kNSH; ++q) dx[q / kNSH][q % kNSH] = make_float2(0.0f, 0.0f);
    symcon_backward_group<LOUT, PARTS>(part, x, coef + (long long)species[lead] * SymconShape<LOUT>::kTerms * kC + c, g, dx);
    add_parts<kNSH, PARTS, CH>(dx, part, t, shared);
    if (part == 0) store_pairs(d_msg, atom, c, dx);
}

// h[a][k][c] = table[species[a]][k][c]  (layer 0's species-only skip connection)
__global__ void k_fill_from_species(int n_atoms, int row, const int32_t* __restrict__ species,
                                    const float* __restrict__ table, float* __restrict__ out) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= (long long)n_atoms * row) return;
    const int a = (int)(i / row), k = (int)(i % row);
    out[i] = table[(long long)species[a] * row + k];
}

// One warp per atom. Non-last layers: e += h[a][0][:] . w, gradient w. Last layer: 128 -> 16 -> SiLU -> 1 with its
// gradient. The energy scale is folded in here. mode bit 0: add to node_energy instead of overwriting.
__global__ void __launch_bounds__(128)
k_readout(int n_atoms, int n_energy, int dim_first, int dim_last, int mlp_hidden, float scale, float shift, float silu_norm,
          const float* __restrict__ h_first, const float* __restrict__ h_last, const float* __restrict__ w_first,
          const float* __restrict__ w_last0, const float* __restrict__ w_last1, float* __restrict__ node_energy,
          float* __restrict__ d_h_first, float* __restrict__ d_h_last) {
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int a = blockIdx.x * 4 + warp;
    if (a >= n_atoms) return;
    if (a >= n_energy) {
        // an atom whose energy belongs to another domain: it contributes no energy and seeds no gradient
        float* df = d_h_first + (long long)a * dim_first * kC;
        for (int k = lane; k < dim_first * kC; k += 32) df[k] = 0.0f;
        if (lane == 0) node_energy[a] = 0.0f;
        return;
    }
    // first readout (linear) and the gradient it leaves on h_first's scalars; other components start at zero
    float e = 0.0f;
    const float* hf = h_first + (long long)a * dim_first * kC;
    float* df = d_h_first + (long long)a * dim_first * kC;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int c = lane + 32 * q;
        e = fmaf(hf[c], w_first[c], e);
        df[c] = scale * w_first[c];
    }
    for (int k = kC + lane; k < dim_first * kC; k += 32) df[k] = 0.0f;
    // last readout
    const float* hl = h_last + (long long)a * dim_last * kC;
    float z[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) z[j] = 0.0f;
    float hv[4];
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int c = lane + 32 * q;
        hv[q] = hl[c];
#pragma unroll
        for (int j = 0; j < 16; ++j) z[j] = fmaf(hv[q], w_last0[c * 16 + j], z[j]);
    }
    float dz[16];
#pragma unroll
    for (int j = 0; j < 16; ++j) {
        const float zz = warp_sum(z[j]);
        const float sig = 1.0f / (1.0f + expf(-zz));
        e += (lane == 0) ? silu_norm * zz * sig * w_last1[j] : 0.0f;
        dz[j] = scale * w_last1[j] * silu_norm * sig * (1.0f + zz * (1.0f - sig));
    }
    e = warp_sum(e);
    if (lane == 0) node_energy[a] = scale * e + shift;
    float* dl = d_h_last + (long long)a * dim_last * kC;
#pragma unroll
    for (int q = 0; q < 4; ++q) {
        const int c = lane + 32 * q;
        float g = 0.0f;
#pragma unroll
        for (int j = 0; j < 16; ++j) g = fmaf(w_last0[c * 16 + j], dz[j], g);
        dl[c] = g;
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

namespace {

template <int LOUT, int PARTS, int CH, int MINB>
int launch_forward_group(int n_rows, int n_groups, const float* coef, const int32_t* species, const int32_t* groups,
                         const float* msg, float* basis, cudaStream_t stream) {
    constexpr int smem = (PARTS / 2) * 2 * SymconShape<LOUT>::kOut * CH * (int)sizeof(float2);
    auto kernel = k_symcon_forward_group<LOUT, PARTS, CH, MINB>;
    kernel<<<n_groups * (kC / CH), CH * PARTS, smem, stream>>>(n_rows, coef, species, groups, msg, basis);
    return FMB_OK;
}

template <int LOUT, int PARTS, int CH, int MINB>
int launch_backward_group(int n_rows, int n_groups, const float* coef, const int32_t* species, const int32_t* groups,
                          const float* msg, const float* d_basis, float* d_msg, cudaStream_t stream) {
    constexpr int smem = (PARTS / 2) * 2 * kNSH * CH * (int)sizeof(float2);
    auto kernel = k_symcon_backward_group<LOUT, PARTS, CH, MINB>;
    kernel<<<n_groups * (kC / CH), CH * PARTS, smem, stream>>>(n_rows, coef, species, groups, msg, d_basis, d_msg);
    return FMB_OK;
}

// Few groups leave SMs without work and each thread with a chain of 94, 410 or 887 terms: two sets of threads share the
// monomials (249 atoms, both layers: 28 -> 18 us forward, 36 -> 23 us adjoint). With more groups one set does, since the
// second one's inputs and sums cost more than the shorter chain gives (10,368 atoms: 83 against 99 us forward).
constexpr int kFewGroups = 148;

template <int LOUT>
int symcon_forward_launch(int n_rows, int n_groups, const float* coef, const int32_t* species, const int32_t* groups,
                          const float* msg, float* basis, cudaStream_t stream) {
    if (n_groups <= kFewGroups) return launch_forward_group<LOUT, 2, 64, 1>(n_rows, n_groups, coef, species, groups, msg, basis, stream);
    return launch_forward_group<LOUT, 1, 64, 1>(n_rows, n_groups, coef, species, groups, msg, basis, stream);
}

// The adjoint holds the messages of four atoms and their gradients (170 registers, 234 for outputs up to l = 2): CTAs of
// one warp fill the registers of an SM evenly (486 groups of the 1,944-atom cell in CTAs of four are a wave and a tenth:
// 55 us, 48 with single warps, 148 against 168 us at 10,368 atoms); for l = 2 whole CTAs read the coefficients together
// (13,824 atoms: 294 us, 384 with single warps).
template <int LOUT>
int symcon_backward_launch(int n_rows, int n_groups, const float* coef, const int32_t* species, const int32_t* groups,
                           const float* msg, const float* d_basis, float* d_msg, cudaStream_t stream) {
    if (n_groups <= kFewGroups)
        return launch_backward_group<LOUT, 2, 64, 1>(n_rows, n_groups, coef, species, groups, msg, d_basis, d_msg, stream);
    if constexpr (LOUT == 2)
        return launch_backward_group<LOUT, 1, 128, 1>(n_rows, n_groups, coef, species, groups, msg, d_basis, d_msg, stream);
    else
        return launch_backward_group<LOUT, 1, 32, 12>(n_rows, n_groups, coef, species, groups, msg, d_basis, d_msg, stream);
}

}  // namespace

#define FMB_TRY_SYM(expr)        \
    {                            \
        const int rc__ = (expr); \
        if (rc__) return rc__;   \
    }

int symcon_forward(int n_atoms, int n_terms, int out_dim, const int32_t* terms, const float* coef,
                   const int32_t* species, const float* msg, float* basis, const int32_t* groups, int n_groups,
                   cudaStream_t stream) {
    (void)terms;
    if (n_atoms <= 0) return FMB_OK;
#define FMB_SYM(L_)                                                                                              \
    {                                                                                                            \
        FMB_REQUIRE(n_terms == SymconShape<L_>::kTerms, "symcon: coefficient table does not match the kernel"); \
        if (groups && n_groups > 0)                                                                              \
            FMB_TRY_SYM((symcon_forward_launch<L_>(n_atoms, n_groups, coef, species, groups, msg, basis, stream)))  \
        else                                                                                                     \
            k_symcon_forward<L_><<<n_atoms, kC, 0, stream>>>(n_atoms, n_terms, coef, species, msg, basis);       \
    }
    if (out_dim == 1) FMB_SYM(0) else if (out_dim == 4) FMB_SYM(1) else if (out_dim == 9) FMB_SYM(2) else {
        FMB_REQUIRE(false, "symcon: unsupported output irreps");
    }
#undef FMB_SYM
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

int symcon_backward(int n_atoms, int n_terms, int out_dim, const int32_t* terms, const float* coef,
                    const int32_t* species, const float* msg, const float* d_basis, float* d_msg, const int32_t* groups,
                    int n_groups, cudaStream_t stream) {
    (void)terms;
    if (n_atoms <= 0) return FMB_OK;
#define FMB_SYM(L_)                                                                                                  \
    {                                                                                                                \
        FMB_REQUIRE(n_terms == SymconShape<L_>::kTerms, "symcon: coefficient table does not match the kernel");     \
        if (groups && n_groups > 0)                                                                                  \
            FMB_TRY_SYM((symcon_backward_launch<L_>(n_atoms, n_groups, coef, species, groups, msg, d_basis, d_msg, stream))) \
        else                                                                                                         \
            k_symcon_backward<L_><<<n_atoms, kC, 0, stream>>>(n_atoms, n_terms, coef, species, msg, d_basis, d_msg); \
    }
    if (out_dim == 1) FMB_SYM(0) else if (out_dim == 4) FMB_SYM(1) else if (out_dim == 9) FMB_SYM(2) else {
        FMB_REQUIRE(false, "symcon: unsupported output irreps");
    }
#undef FMB_SYM
    FMB_LAUNCH_CHECK();
    return FMB_OK;
}

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
    k_readout<<<ceil_div(n_atoms, 4), 128, 0, stream>>>(n_atoms, n_energy, dim_first, dim_last, m->mlp_hidden, m->scale, m->shift,
                                                        m->silu_norm, h_first, h_last, m->layer[0].w_readout, w_last,
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
