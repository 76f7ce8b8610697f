// Symmetric contraction, adjoint (see symcon.cuh).

#include "symcon.cuh"

namespace fmb {

namespace {

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

template <int LOUT, int PARTS, int CH, int MINB>
int launch_backward_group(int n_rows, int n_groups, const float* coef, const int32_t* species, const int32_t* groups,
                          const float* msg, const float* d_basis, float* d_msg, cudaStream_t stream) {
    constexpr int smem = (PARTS / 2) * 2 * kNSH * CH * (int)sizeof(float2);
    auto kernel = k_symcon_backward_group<LOUT, PARTS, CH, MINB>;
    kernel<<<n_groups * (kC / CH), CH * PARTS, smem, stream>>>(n_rows, coef, species, groups, msg, d_basis, d_msg);
    return FMB_OK;
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

}  // namespace fmb
