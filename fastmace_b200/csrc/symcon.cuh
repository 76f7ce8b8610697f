// Symmetric contraction (correlation 3) as a species-dependent polynomial in the 16 message components: what the forward
// kernels (symcon_forward.cu) and the adjoint (symcon_backward.cu) share. The generated bodies take a minute to compile, so
// the two stand in translation units of their own.
//
// Reference: EquivariantProductBasisBlock / SymmetricContraction of mace-torch, in the polynomial form the reference's
// generated kernels evaluate (fastmace/kernels/cuda/sc_generated.py:1-20: one block per atom, one thread per
// channel, y_C = sum_a w_a sum coef * monomial).
//
// One thread per (atom, channel); the polynomial is generated straight-line code (generated/symcon_generated.cuh):
// 16 inputs and the outputs live in registers, each coefficient is one coalesced load from the [species][term][C] table.
//
// The same for the four atoms of a group (one species; -1 = empty slot; atoms at or beyond n_rows are skipped): a
// coefficient is loaded once and used for two pairs of atoms on the packed FP32 pipe. A CTA takes CH of the 128 channels;
// PARTS sets of CH threads share them, each with a run of the monomials, and their sums meet in shared memory.
//
// Bound: the coefficient table that a group streams from L2 (48, 210 or 454 KB for outputs up to l = 0, 1, 2), and with few
// groups the chain of a thread's terms. Two atoms at a time on scalar instructions, as before: 1,944 atoms 41 -> 31 us
// forward (both layers), 10,368 atoms 117 -> 83 and 170 -> 148 us, 13,824 atoms of the large model 445 -> 183 and
// 364 -> 294 us.
#pragma once

#include "stages.cuh"
#include "generated/symcon_generated.cuh"

namespace fmb {

namespace {

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

// Few groups leave SMs without work and each thread with a chain of 94, 410 or 887 terms: two sets of threads share the
// monomials (249 atoms, both layers: 28 -> 18 us forward, 36 -> 23 us adjoint). With more groups one set does, since the
// second one's inputs and sums cost more than the shorter chain gives (10,368 atoms: 83 against 99 us forward).
constexpr int kFewGroups = 148;

}  // namespace

#define FMB_TRY_SYM(expr)        \
    {                            \
        const int rc__ = (expr); \
        if (rc__) return rc__;   \
    }

}  // namespace fmb
