// h3g_eigen.cu — the main engine's model eigensystems on the device.
//
// For every model k of an installed model table: A = D^1/2 Q_k D^-1/2 with D = diag(pi) (pi
// floored at 1e-12), its symmetric part, diagonalised by the parallel cyclic Jacobi of
// h3g_jacobi.cuh; lambda clamped to <= 0; U_pi = D^-1/2 E and V_pi = E^T D^1/2.  This is the
// reference's MG94Matrix::update eigen step (rate_matrix.hpp:229-249, Eigen's
// SelfAdjointEigenSolver there).  The outputs are the engine's padded 64 x 64 layouts (lam, U,
// U^T, V); padding states stay decoupled (zero coupling, eigenvalue 0, zero rows and columns of
// U and V), so they add nothing to P(t) = U diag(e^{lambda t}) V.
#include "h3g_common.cuh"
#include "h3g_jacobi.cuh"
#include "h3g_kernels.h"

namespace h3g {

namespace {

constexpr int kET = jac::kThreads;
constexpr int kEigMaxSweeps = 30;

// grid (nmod), block kET: one model per CTA.  kSym: by the sweeps on half of the matrix (265 us instead of 398 us).  They are
// as accurate, but not the same bits, and a gradient over branches far shorter than the changes on them amplifies the last bits
// of an eigensystem by 1e6 and more; so the FP64 path keeps the rotations it has always had, and the mixed path takes the
// faster ones.  Random codons over branches of 1e-8 to 1e-4, against an 80-bit series: site log-likelihoods off by 2e-4 (1e-4),
// 1 to 17 (1e-6) and 60 (1e-8) with either, whichever is the closer; from 1e-2 on the mixed path's own rounding is all there is.
template <bool kSym>
__global__ void __launch_bounds__(kET) k_model_eig(const double* __restrict__ Q, const double* __restrict__ pi, int S,
                                                   double* lam, double* U, double* UT, double* V) {
    pdl_enter();
    extern __shared__ __align__(16) double sm[];
    constexpr int LD = jac::LD;
    double* A = sm;
    double* E = sm + SP * LD;
    __shared__ double sq[SP], isq[SP];
    __shared__ jac::Scratch js;
    const int tid = threadIdx.x, k = blockIdx.x;
    const double* Qk = Q + size_t(k) * SP2;
    if (tid < SP) {
        const double r = tid < S ? sqrt(fmax(pi[tid], 1e-12)) : 0.0;
        sq[tid] = r;
        isq[tid] = tid < S ? 1.0 / r : 0.0;
    }
    __syncthreads();
    for (int e = tid; e < SP2; e += kET) {
        const int i = e >> 6, j = e & 63;
        A[i * LD + j] = (i < S && j < S) ? sq[i] * Qk[e] * isq[j] : 0.0;
        E[i * LD + j] = i == j ? 1.0 : 0.0;
    }
    __syncthreads();
    for (int e = tid; e < SP2; e += kET) {            // symmetric part (rate_matrix.hpp:236-237)
        const int i = e >> 6, j = e & 63;
        if (i < j) {
            const double m = 0.5 * (A[i * LD + j] + A[j * LD + i]);
            A[i * LD + j] = m;
            A[j * LD + i] = m;
        }
    }
    __syncthreads();
    if constexpr (kSym) jac::sweeps_sym(sm, js, kEigMaxSweeps);
    else jac::sweeps(sm, js, kEigMaxSweeps);
    double* lk = lam + size_t(k) * SP;
    double* Uk = U + size_t(k) * SP2;
    double* UTk = UT + size_t(k) * SP2;
    double* Vk = V + size_t(k) * SP2;
    if (tid < SP) lk[tid] = tid < S ? fmin(js.lam[tid], 0.0) : 0.0;
    for (int e = tid; e < SP2; e += kET) {
        const int a = e >> 6, b = e & 63;
        const bool real = a < S && b < S;
        const double u = real ? isq[a] * E[a * LD + b] : 0.0;     // U_pi[i = a][k = b]
        Uk[e] = u;
        UTk[size_t(b) * SP + a] = u;
        Vk[e] = real ? E[b * LD + a] * sq[b] : 0.0;                // V_pi[k = a][j = b]
    }
}

// A model's arrays from the caller's layout in pinned host memory to the engine's: matrices S x S to 64 x 64, padded with
// zeros, and transposed where asked (a CTA each), vectors and byte arrays by the last CTA.  Read over the bus once,
// coalesced; padding and transposing on the host and copying from pageable memory took 350 us for 3 codon models with
// 8 directions, and this kernel takes about the bus time of the unpadded arrays.
__global__ void __launch_bounds__(256) k_model_install(ModelInstall in) {
    pdl_enter();
    const int tid = threadIdx.x, S = in.S;
    int b = blockIdx.x;
    for (int g = 0; g < in.n_mat; b -= in.mat[g].count, ++g) {
        if (b >= in.mat[g].count) continue;
        __shared__ double tile[SP * (SP + 1)];
        const double* src = in.mat[g].src + size_t(b) * S * S;
        double* dst = in.mat[g].dst + size_t(b) * SP2;
        for (int e = tid; e < SP * (SP + 1); e += 256) tile[e] = 0.0;
        __syncthreads();
#pragma unroll 8
        for (int e = tid; e < S * S; e += 256) tile[(e / S) * (SP + 1) + e % S] = src[e];
        __syncthreads();
        for (int e = tid; e < SP2; e += 256) dst[e] = tile[(e >> 6) * (SP + 1) + (e & 63)];
        if (double* dt = in.mat[g].dst_t)
            for (int e = tid; e < SP2; e += 256) dt[size_t(b) * SP2 + e] = tile[(e & 63) * (SP + 1) + (e >> 6)];
        return;
    }
    for (int g = 0; g < in.n_vec; ++g) {
        const auto& v = in.vec[g];
        for (int e = tid; e < v.rows * v.pad; e += 256) {
            const int r = e / v.pad, c = e % v.pad;
            v.dst[e] = c < v.width ? v.src[r * v.width + c] : 0.0;
        }
    }
}

}  // namespace

int launch_model_install(const ModelInstall& in, cudaStream_t s) {
    int blocks = in.n_vec ? 1 : 0;
    for (int g = 0; g < in.n_mat; ++g) blocks += in.mat[g].count;
    launch_k(k_model_install, blocks, 256, 0, s, in);
    return 1;
}

void eigen_configure() {
    cudaFuncSetAttribute(k_model_eig<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(jac::kSmem));
    cudaFuncSetAttribute(k_model_eig<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(jac::kSymSmem));
}

int launch_model_eig(const double* Q, const double* pi, int S, int nmod, double* lam, double* U, double* UT, double* V,
                     bool mixed, cudaStream_t s) {
    if (mixed) launch_k(k_model_eig<true>, nmod, kET, jac::kSymSmem, s, Q, pi, S, lam, U, UT, V);
    else launch_k(k_model_eig<false>, nmod, kET, jac::kSmem, s, Q, pi, S, lam, U, UT, V);
    return 1;
}

}  // namespace h3g
