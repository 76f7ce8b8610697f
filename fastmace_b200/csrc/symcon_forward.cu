// Symmetric contraction, forward (see symcon.cuh).

#include "symcon.cuh"

namespace fmb {

namespace {

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
int launch_forward_group(int n_rows, int n_groups, const float* coef, const int32_t* species, const int32_t* groups,
                         const float* msg, float* basis, cudaStream_t stream) {
    constexpr int smem = (PARTS / 2) * 2 * SymconShape<LOUT>::kOut * CH * (int)sizeof(float2);
    auto kernel = k_symcon_forward_group<LOUT, PARTS, CH, MINB>;
    kernel<<<n_groups * (kC / CH), CH * PARTS, smem, stream>>>(n_rows, coef, species, groups, msg, basis);
    return FMB_OK;
}

template <int LOUT>
int symcon_forward_launch(int n_rows, int n_groups, const float* coef, const int32_t* species, const int32_t* groups,
                          const float* msg, float* basis, cudaStream_t stream) {
    if (n_groups <= kFewGroups) return launch_forward_group<LOUT, 2, 64, 1>(n_rows, n_groups, coef, species, groups, msg, basis, stream);
    return launch_forward_group<LOUT, 1, 64, 1>(n_rows, n_groups, coef, species, groups, msg, basis, stream);
}

}  // namespace

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

}  // namespace fmb
