// Internal launch functions shared between the translation units of libfmb200.
#pragma once

#include "fmb_common.cuh"

namespace fmb {

// `count`: device edge count to featurise (null = the list's own count)
int edge_features(const fmb_model_t* model, const fmb_nl_t* nl, const fmb_work_t* work, const double* positions,
                  const long long* count, cudaStream_t stream);

struct TpArgs {
    int lin;
    bool species_x;
    int n_atoms;           // atoms of the list (rows of row_ptr)
    int n_rows;            // receivers this launch computes: [0, n_rows)
    int n_valid;           // backward: atoms [0, n_valid) have a message gradient, the others read as zero
    int fresh_from;        // backward: atoms at or beyond this start their force / virial sums from zero
    long long chunk_e0, chunk_edges, tangent_offset;
    bool whole_list;       // the launch covers the whole edge list (one chunk)
    const long long* count;
    const int32_t* row_ptr;
    const int32_t* senders;
    const int32_t* species;
    const float* x;
    const float* edge_sh;
    const float* edge_vec;
    const float* tp_w;
    float* mid;            // forward output
    const float* d_mid;    // backward input
    float* d_x;
    float* force_acc;
    float* atom_virial;
    int first_layer_of_pass;
    uint32_t* error_word;  // device status word for bounded-wait failures of the staged kernels
    const int32_t* slot;   // or null: the weights of edge e are row slot[e] of tp_w (one row per pair of opposite edges)
};
int tp_forward_launch(const TpArgs& t, cudaStream_t stream);
int tp_backward_launch(const TpArgs& t, cudaStream_t stream);
// senders with rows of their own (tp_coupled.cu)
int tp_forward_coupled_launch(const TpArgs& t, cudaStream_t stream);

// Per-edge radial weights (or their d/dr) [rows][n_paths * 128] = hidden [rows][64] x last radial layer on the
// tensor cores (radial_weights.cu); FMB_ERR_UNSUPPORTED without the weight image.
// `row_index` (or null): output row r is computed from hidden row row_index[r]
int radial_weights_tc(const float* hidden, const float* image, float* out, int rows, int n_paths, const long long* limit,
                      long long limit_offset, const int32_t* row_index, uint32_t* error_word, int max_ctas,
                      cudaStream_t stream);

// first layer in reassociated form (outer products per receiver and sender species)
struct FirstArgs {
    int n_rows, n_valid, fresh_from, n_species;
    const long long* count;
    const int32_t* row_ptr;
    const int32_t* senders;
    const int32_t* species;
    const float* edge_sh;
    const float* edge_vec;
    const float* hidden;           // [edges][64] last hidden radial layer of the first interaction
    const float* hidden_tangent;   // its derivative with respect to the edge length
    float* s;                      // forward output [n][16][n_species][64]
    const float* d_s;              // backward input, same layout
    float* force_acc;
    float* atom_virial;
    int first_layer_of_pass;
};
int first_accumulate_launch(const FirstArgs& f, cudaStream_t stream);
int first_backward_launch(const FirstArgs& f, cudaStream_t stream);

// Adjoint with per-edge hand-over (adjoint_edges.cu)
struct EdgeAdjointArgs {
    int lin;
    int n_atoms;           // atoms of the list
    int n_rows;            // receivers [0, n_rows)
    int n_valid;           // atoms [0, n_valid) have a message gradient
    int n_gather;          // atoms [0, n_gather) collect the gradient of their own features (d_x rows)
    long long chunk_e0, chunk_edges;   // this launch covers the edges [chunk_e0, chunk_e0 + chunk_edges) below the count
    const long long* count;
    const int32_t* row_ptr;
    const int32_t* senders;
    const int32_t* receivers;
    const int32_t* mirror;
    const float* x;
    const float* edge_sh;
    const float* edge_vec;
    const float* tp_w;             // [chunk edges][paths * C] values, d/dr behind them at tangent_offset
    long long tangent_offset;
    const float* d_mid;
    float* dxe;                    // [edges from dx_e0 on][(lin + 1)^2][C]
    long long dx_e0, dx_rows;      // first edge and rows of dxe
    float* qe;                     // [edges][4]
    float* d_x;                    // [n_rows][(lin + 1)^2][C]
    uint32_t* error_word;
    const int32_t* slot;           // or null: the weights of edge e are row slot[e] of tp_w
};
// Interactions after the first with the last radial layer inside the kernel (tp_onchip.cu; node l_max 1)
struct TpOnChipArgs {
    int lin, n_rows;
    const int32_t* row_ptr;
    const int32_t* senders;
    const float* x;
    const float* edge_sh;
    const float* edge_vec;
    const float* hidden;           // [edges][64]
    const float* tangent;
    const float* image;            // the last radial layer, behind the producer's image in fmb_layer_t.rad_img
    float* mid;                    // forward output
    const float* d_mid;            // adjoint input
    long long e0, e_span;          // adjoint: the edges [e0, e0 + e_span) below the count
    float* dxe;                    // [edges from dx0 on][(lin + 1)^2][C]
    long long dx0;
    // forward: sums of rows that lie in several ranges of edges; adjoint output: per half of the channels and edge the
    // gradients of the 16 harmonics and of the length, [2][part_stride][20], to be added up
    float* scratch;
    long long part_stride;
    uint32_t* error_word;
};
// floats of `scratch` for a list of `edges` edges (negative: no kernel for this node l_max)
long long tp_onchip_scratch_floats(int lin, long long edges);
// of them the adjoint's output
constexpr long long tp_onchip_part_floats(long long edges) { return 2 * edges * 20; }
int tp_forward_onchip(const TpOnChipArgs& t, cudaStream_t stream);
int tp_adjoint_onchip(const TpOnChipArgs& t, cudaStream_t stream);

// `slot`, `list`, `list_count` (or null): the edges below *listed_below that stand for their pair
int mirror_map(const fmb_nl_t* nl, int32_t* mirror, uint32_t* status, const long long* listed_below, int32_t* slot,
               int32_t* list, long long* list_count, int list_capacity, cudaStream_t stream);
// per-edge adjoint of an interaction after the first for one chunk of edges
int tp_adjoint_edges(const EdgeAdjointArgs& t, cudaStream_t stream);
// its form where every row carries a gradient (tp_coupled.cu)
int tp_adjoint_coupled_launch(const EdgeAdjointArgs& t, cudaStream_t stream);
// the gather of the sender-side gradients into d_x: of the whole list after its last chunk, or (`chunk`: dxe holds one
// chunk) behind every chunk, the first of which starts d_x from zero
int gather_sender_gradient(const EdgeAdjointArgs& t, bool chunk, cudaStream_t stream);
// first interaction: adds its edge-vector gradients to qe (rows below n_add) or stores them; with `parts` it adds the later
// interaction's gradients of harmonics and length, parts[2][part_stride][20], to its own before they become one of the edge
// vector, and what qe holds is not read
int first_adjoint_edges(const FirstArgs& f, int n_add, float* qe, const float* parts, long long part_stride, cudaStream_t stream);
// forces (as gradients) and per-atom virials from the per-edge gradients; only the edges into atoms [0, n_valid) carry
// a gradient (the others are read as zero, whatever qe holds for them)
int force_gather(int n_atoms, int n_valid, const int32_t* row_ptr, const int32_t* senders, const int32_t* mirror,
                 const float* qe, const float* edge_vec, float* force_acc, float* atom_virial, cudaStream_t stream);

int symcon_forward(int n_atoms, int n_terms, int out_dim, const int32_t* terms, const float* coef,
                   const int32_t* species, const float* msg, float* basis, const int32_t* groups, int n_groups,
                   cudaStream_t stream);
int symcon_backward(int n_atoms, int n_terms, int out_dim, const int32_t* terms, const float* coef,
                    const int32_t* species, const float* msg, const float* d_basis, float* d_msg, const int32_t* groups,
                    int n_groups, cudaStream_t stream);
int fill_from_species(int n_atoms, int row, const int32_t* species, const float* table, float* out, cudaStream_t stream);
int readout(const fmb_model_t* m, int n_atoms, int n_energy, const float* h_first, const float* h_last, float* node_energy,
            float* d_h_first, float* d_h_last, cudaStream_t stream);
int reduce_outputs(const fmb_model_t* m, const fmb_work_t* w, int n_energy, double volume, cudaStream_t stream);
int commit_forces(const fmb_work_t* w, double* f64, double* e64, double* s64, cudaStream_t stream);

}  // namespace fmb
