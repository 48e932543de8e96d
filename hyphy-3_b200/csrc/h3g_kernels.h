// h3g_kernels.h — host-callable launchers of the device pipeline (one per stage).
// Each returns the number of kernels it enqueued on the stream.
#pragma once
#include "h3g_common.cuh"

namespace h3g {

// Arrays of a model in pinned host memory and where the engine wants them (k_model_install).
struct ModelInstall {
    struct Mat { const double* src; double* dst; double* dst_t; int count; } mat[3];       // [count][S][S] -> [count][64][64]
    struct Vec { const double* src; double* dst; int rows, width, pad; } vec[9];           // [rows][width] -> [rows][pad], 8-byte words
    int n_mat, n_vec, S;
};
int launch_model_install(const ModelInstall& in, cudaStream_t s);

void fp64_configure();
int launch_build_P(const Topo& t, const Model& md, const Work& w, cudaStream_t s);
int launch_prep_given_P(const Topo& t, const Work& w, cudaStream_t s);
int launch_inside_fp64(const Topo& t, const Model& md, const Work& w, const int* d_nodes, int count, cudaStream_t s);
int launch_root(const Topo& t, const Model& md, const Work& w, cudaStream_t s);
// d_kids: internal children of one depth's nodes
int launch_outside_fp64(const Topo& t, const Model& md, const Work& w, const int* d_kids, int count, cudaStream_t s);
// A of the listed internal branches, and of leaves: n_leaves entries of one leaf (y = -1) or the two of a two-leaf node,
// then n_many leaves of nodes with more than kFewKids children
constexpr int kFewKids = 9;
int launch_accumA_fp64(const Topo& t, const Model& md, const Work& w, const int* d_internal, int n_internal, const int2* d_leaves,
                       int n_leaves, int n_many, cudaStream_t s);
// The same passes for t.S <= kFewStates, one launch each (h3g_few.cu)
int launch_inside_few(const Topo& t, const Model& md, const Work& w, cudaStream_t s);
int launch_outside_few(const Topo& t, const Model& md, const Work& w, cudaStream_t s);
int launch_accumA_few(const Topo& t, const Model& md, const Work& w, cudaStream_t s);
int launch_frechet(const Topo& t, const Model& md, const Work& w, int want_global, cudaStream_t s);
int launch_global(const Topo& t, const Model& md, const Work& w, cudaStream_t s);
int launch_dir(const Topo& t, const Model& md, const Work& w, cudaStream_t s);
int launch_small(const Topo& t, const Model& md, const Work& w, int grads, cudaStream_t s);
void eigen_configure();
// Model eigensystems on the device (h3g_eigen.cu): Q [nmod][64*64] padded, pi [64] -> lam, U, U^T, V.
int launch_model_eig(const double* Q, const double* pi, int S, int nmod, double* lam, double* U, double* UT, double* V,
                     bool mixed, cudaStream_t s);
int launch_pack_result(const Topo& t, const Model& md, const Work& w, int grads, int global, double* dst, cudaStream_t s);

}  // namespace h3g
