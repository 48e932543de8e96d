// h3g_fp64.cu — FP64 kernels of the likelihood + adjoint-gradient pipeline.
//
// Per evaluation (one CUDA stream, level-synchronous over the tree):
//   k_build_P      P_{m,b} = sum_k c_k clamp(U_k diag(e^{lam_k tau}) V_k), dP = d P / d t
//                  (rate_matrix.hpp:251-257, likelihood.hpp:1118-1127, busted.hpp:1191-1216),
//                  FP64 tensor-core products
//   k_inside       one launch per height level: D_u = prod_c P_c D_c with power-of-two
//                  rescaling, then the message P_u D_u for the parent (likelihood.hpp:500-597)
//   k_root         L = pi . D_root, log-sum-exp over rate classes, per-pattern scale
//                  factors f = w * post / L (likelihood.hpp:599-610, busted.hpp:1346-1375)
//   k_outside      one launch per depth level, internal children: V_c = 2^{e_u} U_u o prod_{s != c} P_s D_s,
//                  U_c = P_c^T V_c (likelihood.hpp:612-761)
//   k_accumA_int, k_accumA_leaf   A_{m,b} = sum_p f V D^T  (likelihood.hpp:1435 generalised)
//   k_frechet      dlnL/dt_b = <A, dP>; spectral Frechet pieces U^T A V^T o E
//                  (likelihood.hpp:1428-1471)
//   k_hsum, k_dir, k_small   fixed-order reductions -> lnL, gradients
// All reductions run in a fixed order, so repeated evaluations are bit-identical.
#include <algorithm>
#include <climits>
#include <cstdlib>
#include "h3g_common.cuh"
#include "h3g_kernels.h"
#include "h3g_mixed.h"
#include "h3g_tc.cuh"

namespace h3g {

__device__ __forceinline__ void stage_matrix(double* __restrict__ s, const double* __restrict__ g, int tid, int nthr) {
    const double2* g2 = reinterpret_cast<const double2*>(g);
    double2* s2 = reinterpret_cast<double2*>(s);
    for (int k = tid; k < SP2 / 2; k += nthr) s2[k] = __ldg(g2 + k);
}

// --------------------------------------------------- FP64 tensor-core products
// 64x64x64 products on the FP64 tensor cores (mma.sync m8n8k4 .f64; tcgen05 has no FP64
// kind) by the 8 warps of a 256-thread CTA: warp w owns rows 16(w/2) .. +16 and columns
// 32(w%2) .. +32 as 2 x 4 tiles of 8x8, operands and results stay in registers between
// the k steps.  Both operands are row-major in shared memory with a padded stride of 68
// doubles: the fragment loads of a half-warp, (row + lane/4) * 68 + k + lane%4 and
// (k + lane%4) * 68 + col + lane/4, fall in 16 different banks.
constexpr int LDM = SP + 4;

struct Frag64 {
    double v[2][4][2];        // C[r0 + 8i + lane/4][c0 + 8j + 2(lane%4) + e]
};

__device__ __forceinline__ void frag_zero(Frag64& f) {
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j) f.v[i][j][0] = f.v[i][j][1] = 0.0;
}
// position of f.v[i][j][e] in the 64x64 result
__device__ __forceinline__ int frag_row(int i) { return 16 * (int(threadIdx.x) >> 6) + 8 * i + ((threadIdx.x & 31) >> 2); }
__device__ __forceinline__ int frag_col(int j, int e) {
    return 32 * ((int(threadIdx.x) >> 5) & 1) + 8 * j + 2 * (threadIdx.x & 3) + e;
}

__device__ __forceinline__ void dmma(double& d0, double& d1, double a, double b) {
    asm("mma.sync.aligned.m8n8k4.row.col.f64.f64.f64.f64 {%0, %1}, {%2}, {%3}, {%0, %1};"
        : "+d"(d0), "+d"(d1)
        : "d"(a), "d"(b));
}

// c = X Y, X and Y [64][LDM] in shared memory
__device__ __forceinline__ void mm64(const double* __restrict__ X, const double* __restrict__ Y, Frag64& c) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const int r0 = 16 * (wp >> 1), c0 = 32 * (wp & 1), g = lane >> 2, q = lane & 3;
    frag_zero(c);
#pragma unroll 4
    for (int k = 0; k < SP; k += 4) {
        double a[2], b[4];
#pragma unroll
        for (int i = 0; i < 2; ++i) a[i] = X[(r0 + 8 * i + g) * LDM + k + q];
#pragma unroll
        for (int j = 0; j < 4; ++j) b[j] = Y[(k + q) * LDM + c0 + 8 * j + g];
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) dmma(c.v[i][j][0], c.v[i][j][1], a[i], b[j]);
    }
}

// ------------------------------------------------------------------ build P
// grid (n, M): one CTA per branch and rate class computes the whole 64x64
// P_{m,b} = sum_k c_k clamp(U_k diag(e^{lam_k tau}) V_k) and
// dP_{m,b} = sum_k c_k r_m conv_k Q_k clamp(P_k), model by model, as two FP64
// tensor-core products per model (mm64).
// dynamic smem: 2 x 64 x LDM doubles (U e then Q; V then clamp(P_k)).
// kMixed: the split-precision path's operands instead of the FP64 P and P^T, from P staged in
// shared memory: the BF16 hi/mid/lo tiles of P and P^T in the tcgen05 K-major layout (16-byte
// stores of 8 consecutive K), FP32 P^T and the row sums (FP64 and FP32); thread 0 of CTA (0, 0)
// starts the evaluation's epoch of the persistent passes.
template <bool kMixed>
__global__ void __launch_bounds__(256) k_build_P(Topo t, Model md, Work w, MixedWork mw) {
    pdl_enter();
    extern __shared__ __align__(16) double sm[];
    double* sX = sm;                 // U_k diag(e), then Q_k
    double* sY = sm + SP * LDM;      // V_k, then clamp(P_k)
    __shared__ double se[SP];
    __shared__ double srow[2][SP];
    const int b = blockIdx.x, m = blockIdx.y, tid = threadIdx.x;
    if (kMixed && b == 0 && m == 0 && tid == 0) {        // a new evaluation: new epoch, fresh item counters
        mw.sync[0] += 1;
        mw.sync[1] = 0;
        mw.sync[2] = 0;
    }
    if (b == t.root) return;
    const BranchModels bm = branch_models(md, b);
    Frag64 accP, accD;
    frag_zero(accP);
    frag_zero(accD);
    for (int k = bm.k0; k < bm.k1; ++k) {
        const double cw = class_weight(md, bm, k);
        const double cv = time_conv(md, k);
        const double rate = md.rates[m];
        const double tau = rate * w.bl[b] * cv;
        __syncthreads();                          // the previous model's products are done
        if (tid < SP) se[tid] = exp(md.lam[size_t(k) * SP + tid] * tau);
        __syncthreads();
        {
            const double* U = md.U + size_t(k) * SP2;
            const double* V = md.V + size_t(k) * SP2;
            for (int e = tid; e < SP2; e += 256) {
                const int r = e >> 6, l = e & 63;
                sX[r * LDM + l] = __ldg(U + e) * se[l];
                sY[r * LDM + l] = __ldg(V + e);
            }
        }
        __syncthreads();
        Frag64 pk;
        mm64(sX, sY, pk);                         // P_k = (U e) V
        __syncthreads();                          // every warp is done with U e and V
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const double x = fmax(pk.v[i][j][e], 0.0);
                    accP.v[i][j][e] = fma(cw, x, accP.v[i][j][e]);
                    sY[frag_row(i) * LDM + frag_col(j, e)] = x;
                }
        {
            const double* Q = md.Q + size_t(k) * SP2;
            for (int e = tid; e < SP2; e += 256) sX[(e >> 6) * LDM + (e & 63)] = __ldg(Q + e);
        }
        __syncthreads();
        Frag64 qp;
        mm64(sX, sY, qp);                         // Q clamp(P_k)
        const double sc = cw * rate * cv;
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) accD.v[i][j][e] = fma(sc, qp.v[i][j][e], accD.v[i][j][e]);
    }
    const size_t o = mat_off(m, b, t.n);
    if constexpr (!kMixed) {
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int r = frag_row(i), c = frag_col(j, 0);
                *reinterpret_cast<double2*>(w.P + o + r * SP + c) = make_double2(accP.v[i][j][0], accP.v[i][j][1]);
                *reinterpret_cast<double2*>(w.dP + o + r * SP + c) = make_double2(accD.v[i][j][0], accD.v[i][j][1]);
                w.PT[o + c * SP + r] = accP.v[i][j][0];
                w.PT[o + (c + 1) * SP + r] = accP.v[i][j][1];
            }
        // row sums (the message of a leaf without data): the four lanes of a row, then its two column halves
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            double rs = 0.0;
#pragma unroll
            for (int j = 0; j < 4; ++j) rs += accP.v[i][j][0] + accP.v[i][j][1];
            rs += __shfl_xor_sync(0xffffffffu, rs, 1);
            rs += __shfl_xor_sync(0xffffffffu, rs, 2);
            if ((tid & 3) == 0) srow[(tid >> 5) & 1][frag_row(i)] = rs;
        }
        __syncthreads();
        if (tid < SP) w.rs[(size_t(m) * t.n + b) * SP + tid] = srow[0][tid] + srow[1][tid];
    } else {
        __syncthreads();                          // every warp is done reading sX (Q) and sY
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j) {
                const int r = frag_row(i), c = frag_col(j, 0);
                *reinterpret_cast<double2*>(w.dP + o + r * SP + c) = make_double2(accD.v[i][j][0], accD.v[i][j][1]);
                sX[r * LDM + c] = accP.v[i][j][0];
                sX[r * LDM + c + 1] = accP.v[i][j][1];
            }
        __syncthreads();
        // chunk c: row c / 8 of the tile, K = 8 (c % 8) .. +8
        for (int c = tid; c < SP * (SP / 8); c += 256) {
            const int r = c >> 3, k0 = (c & 7) * 8;
            const uint32_t off = tc::kmajor_off16(SP, r, k0) / 2;
            float x[8];
            uint32_t hw[3][4];
            // P tile: row r = output state i, K = input state j
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = float(sX[r * LDM + k0 + e]);
#pragma unroll
            for (int e = 0; e < 4; ++e) tc::split3x2(x[2 * e], x[2 * e + 1], hw[0][e], hw[1][e], hw[2][e]);
#pragma unroll
            for (int q = 0; q < 3; ++q)
                *reinterpret_cast<uint4*>(mw.Bp[q] + o + off) = make_uint4(hw[q][0], hw[q][1], hw[q][2], hw[q][3]);
            // P^T tile: row r = input state j, K = output state i; FP32 P^T row r
#pragma unroll
            for (int e = 0; e < 8; ++e) x[e] = float(sX[(k0 + e) * LDM + r]);
#pragma unroll
            for (int e = 0; e < 4; ++e) tc::split3x2(x[2 * e], x[2 * e + 1], hw[0][e], hw[1][e], hw[2][e]);
#pragma unroll
            for (int q = 0; q < 3; ++q)
                *reinterpret_cast<uint4*>(mw.Bpt[q] + o + off) = make_uint4(hw[q][0], hw[q][1], hw[q][2], hw[q][3]);
            float4* pt = reinterpret_cast<float4*>(mw.PT32 + o + size_t(r) * SP + k0);
            pt[0] = make_float4(x[0], x[1], x[2], x[3]);
            pt[1] = make_float4(x[4], x[5], x[6], x[7]);
        }
        if (tid < SP) {
            double rs = 0.0;
            for (int j = 0; j < SP; ++j) rs += sX[tid * LDM + j];
            w.rs[(size_t(m) * t.n + b) * SP + tid] = rs;
            mw.rs32[(size_t(m) * t.n + b) * SP + tid] = float(rs);
        }
    }
}

// Caller-supplied P (compute_tree_log_likelihood_from_P): derive PT and row sums.
__global__ void k_prep_given_P(Topo t, Work w) {
    pdl_enter();
    const int b = blockIdx.x, tid = threadIdx.x;
    if (b == t.root) return;
    const double* P = w.P + mat_off(0, b, t.n);
    double* PT = w.PT + mat_off(0, b, t.n);
    for (int e = tid; e < SP2; e += blockDim.x) PT[(e % SP) * SP + e / SP] = P[e];
    if (tid < SP) {
        double s = 0.0;
        for (int j = 0; j < SP; ++j) s += P[tid * SP + j];
        w.rs[size_t(b) * SP + tid] = s;
    }
}

// ------------------------------------------------------------------- inside
// CTA = 8 warps x 32 patterns; warp g owns states [8g, 8g+8) of its 32 patterns
// (lane = pattern), so every global access of a partial is a coalesced 256-byte row.
constexpr int kTileP = 32;      // patterns per tile in the FP64 pruning kernels
constexpr int kGroups = 8;      // state groups (warps) per CTA

// The observed state of a child at pattern p (its sense index, or -1; 0 for an internal child, which has none).
__device__ __forceinline__ int child_state(const Topo& t, int2 d, int p) {
    if (d.y <= -2) return 0;
    return d.y < 0 ? -1 : int(t.states[size_t(d.y) * t.Pp + p]);
}
// A child's message for states [8g, 8g+8) of pattern p: the stored message of an internal child; for a leaf in
// state st >= 0 a column of P else the row sums or a masked column sum.
// d: Topo::kdesc entry.
__device__ __forceinline__ void load_msg8(double (&a)[8], const Topo& t, const Work& w, int m, int M, int2 d, int p, int g, int st) {
    if (d.y <= -2) {
        const double* src = w.Ms + part_off(-(d.y + 2), m, M, t.Pp) + size_t(8 * g) * t.Pp + p;
#pragma unroll
        for (int q = 0; q < 8; ++q) a[q] = src[size_t(q) * t.Pp];
        return;
    }
    const double* PTc = w.PT + mat_off(m, d.x, t.n);
    const double* src = PTc + st * SP + 8 * g;
    if (st < 0) {
        const uint64_t mk = d.y < 0 ? t.all_mask : t.masks[size_t(d.y) * t.Pp + p];
        if (mk == 0 || (mk & t.all_mask) == t.all_mask) {
            src = w.rs + (size_t(m) * t.n + d.x) * SP + 8 * g;
        } else {
#pragma unroll
            for (int q = 0; q < 8; ++q) a[q] = 0.0;
            for (uint64_t b = mk; b; b &= b - 1) {
                const double* col = PTc + (__ffsll((long long)b) - 1) * SP + 8 * g;
#pragma unroll
                for (int q = 0; q < 8; ++q) a[q] += __ldg(col + q);
            }
            return;
        }
    }
    const double2* s2 = reinterpret_cast<const double2*>(src);
#pragma unroll
    for (int q = 0; q < 4; ++q) { const double2 x = __ldg(s2 + q); a[2 * q] = x.x; a[2 * q + 1] = x.y; }
}

// Power-of-two renormalisation of a 64-state column spread over the 8 warps:
// returns the shift applied (same on every warp of a lane).
__device__ __forceinline__ int renorm_cols(double (&v)[8], double* smax, int g, int lane) {
    double mx = 0.0;
#pragma unroll
    for (int q = 0; q < 8; ++q) mx = fmax(mx, v[q]);
    smax[g * kTileP + lane] = mx;
    __syncthreads();
    double all = 0.0;
#pragma unroll
    for (int k = 0; k < kGroups; ++k) all = fmax(all, smax[k * kTileP + lane]);
    __syncthreads();
    if (all > 0.0 && all < 0x1p-256) {
        const int sh = -ilogb(all) - 1;
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = ldexp(v[q], sh);
        return sh;
    }
    return 0;
}
// One barrier, a vote: does every thread have a state of 2^-340 or more among its eight?  A column then has a maximum
// of 2^-340 at least and needs no scaling: the product of two such stays far from the end of the range, and
// scaling by powers of two changes no result.  (At 2^-256, the bound of the exchange itself, states 60 powers of
// two below their column's maximum sent most tiles through it.)  Doubles >= 0 compare like the integers of their
// upper words.  S: states; a group beyond them does not count.
__device__ __forceinline__ bool none_small(const double (&v)[8], int g, int S) {
    int hi = 8 * g >= S ? INT_MAX : 0;
#pragma unroll
    for (int q = 0; q < 8; ++q) hi = max(hi, __double2hiint(v[q]));
    return __syncthreads_and(hi >= ((1023 - 340) << 20));
}
// The vote, and the exchange unless it passes.
__device__ __forceinline__ int renorm_if_small(double (&v)[8], double* smax, int g, int lane, int S) {
    return none_small(v, g, S) ? 0 : renorm_cols(v, smax, g, lane);
}

// Partial tiles of the FP64 pruning CTAs in shared memory: [64 states][32 patterns] with a row
// stride of kDL = 36 doubles, so the B-fragment loads (k + lane%4) * 36 + col + lane/4 of a half-warp
// fall in 16 different banks.
constexpr int kDL = kTileP + 4;

__device__ __forceinline__ void cp_async16_f64(double* dst, const double* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;"
                 ::"r"(static_cast<uint32_t>(__cvta_generic_to_shared(dst))), "l"(src) : "memory");
}

// A warp's rows 8g .. 8g+7 of a 64x64 matrix as the A fragments of 16 m8n8k4 products: 16 doubles a thread.
struct RowFrags { double a[SP / 4]; };
__device__ __forceinline__ RowFrags load_rows(const double* __restrict__ mat) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5;
    const double* row = mat + (8 * wp + (lane >> 2)) * SP + (lane & 3);
    RowFrags f;
#pragma unroll
    for (int k = 0; k < SP / 4; ++k) f.a[k] = __ldg(row + 4 * k);
    return f;
}

// dst[i][p] = sum_k M[i][k] sX[k][p] for the CTA's 64 x 32 tile on the FP64 tensor cores
// (mma.sync m8n8k4): warp w owns output rows 8w .. 8w+7 (f), all 32 columns as four 8x8 tiles,
// 16 k steps of 4.  sX [64][kDL]; dst has row stride `stride`
// (state-major partials), each thread storing two adjacent patterns as one 16-byte write.
__device__ __forceinline__ void tile_mm_store(const RowFrags& f, const double* __restrict__ sX, double* __restrict__ dst, size_t stride) {
    const int lane = threadIdx.x & 31, wp = threadIdx.x >> 5, g = lane >> 2, q = lane & 3;
    double c[4][2];
#pragma unroll
    for (int j = 0; j < 4; ++j) c[j][0] = c[j][1] = 0.0;
#pragma unroll
    for (int k = 0; k < SP / 4; ++k) {
        const double* brow = sX + (4 * k + q) * kDL + g;
#pragma unroll
        for (int j = 0; j < 4; ++j) dmma(c[j][0], c[j][1], f.a[k], brow[8 * j]);
    }
    double* d = dst + size_t(8 * wp + g) * stride + 2 * q;
#pragma unroll
    for (int j = 0; j < 4; ++j) *reinterpret_cast<double2*>(d + 8 * j) = make_double2(c[j][0], c[j][1]);
}

// grid (ceil(Pp/32 / tiles), nodes in level, M), block 256: `tiles` pattern tiles of one node and class.  The
// node's matrix stays in registers as fragments for all of them, the next tile's first two messages (and the
// observed states after that) are loaded while this one multiplies, and the rescaling is one vote unless a tile needs it.
// A tile takes about 4600 cycles of an SM, 2048 of them products: the rest is 2500-3600 wavefronts of the L1 (1050
// for each leaf's gathered columns of P, 1024 for the products' B fragments).  1024 taxa x 1200 codons x 4 rates:
// 2.65 ms for all levels; a CTA per tile with the matrix in shared memory and a rescaling exchange per child: 3.40 ms.
// Tried and slower: leaves' matrices staged in shared memory (2.92), columns fetched by cp.async two tiles ahead
// (3.09), whole rows of P^T fetched for leaves (2.93).
__global__ void __launch_bounds__(256, 2) k_inside(Topo t, Model md, Work w, const int* __restrict__ nodes, int tiles) {
    __shared__ __align__(16) double sD[SP * kDL];
    __shared__ double smax[kGroups * kTileP];
    const int u = nodes[blockIdx.y], m = blockIdx.z, tid = threadIdx.x;
    const int g = tid >> 5, lane = tid & 31;
    const int k0 = t.ch_off[u], k1 = t.ch_off[u + 1];
    const int iu = t.iidx[u], M = md.M;
    const size_t Pp = size_t(t.Pp);
    const bool root = (u == t.root), one = k0 < k1, two = k0 + 1 < k1;
    const int t0 = blockIdx.x * tiles, t1 = min(t0 + tiles, t.Pp / kTileP);
    const int2 d0 = one ? t.kdesc[k0] : make_int2(0, -1), d1 = two ? t.kdesc[k0 + 1] : d0;
    double a0[8], a1[8];
    int p = t0 * kTileP + lane;
    int s0 = child_state(t, d0, p), s1 = child_state(t, d1, p);
    pdl_enter();                                                   // above: the problem's tables and patterns only
#pragma unroll
    for (int q = 0; q < 8; ++q) a0[q] = 8 * g + q < t.S ? 1.0 : 0.0;      // a node without children
    if (one) load_msg8(a0, t, w, m, M, d0, p, g, s0);
    if (two) load_msg8(a1, t, w, m, M, d1, p, g, s1);
    RowFrags f;
    if (!root) f = load_rows(w.P + mat_off(m, u, t.n));
    int n0 = 0, n1 = 0;                                            // the next tile's states
    if (t0 + 1 < t1) { n0 = child_state(t, d0, p + kTileP); n1 = child_state(t, d1, p + kTileP); }
    for (int tile = t0; tile < t1; ++tile, p += kTileP) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = two ? a0[q] * a1[q] : a0[q];
        int eown = 0;
        if (!none_small(v, g, t.S)) {                      // (its barrier: the last tile's products are done with sD)
            // the first message by itself, then the product: two columns of a matrix's tiny entries, 2^-537 and
            // below, have a product that is no double
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = a0[q];
            eown = renorm_cols(v, smax, g, lane);
            if (two) {
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] *= a1[q];
                eown += renorm_cols(v, smax, g, lane);
            }
        }
        for (int k = k0 + 2; k < k1; ++k) {
            const int2 d = t.kdesc[k];
            double x[8];
            load_msg8(x, t, w, m, M, d, p, g, child_state(t, d, p));
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] *= x[q];
            eown += renorm_if_small(v, smax, g, lane, t.S);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) sD[(8 * g + q) * kDL + lane] = v[q];
        double* dst = w.D + part_off(iu, m, M, t.Pp) + size_t(8 * g) * Pp + p;
#pragma unroll
        for (int q = 0; q < 8; ++q) dst[q * Pp] = v[q];
        if (g == 0) {
            int ecum = eown;
            for (int k = k0; k < k1; ++k) {
                const int code = t.kdesc[k].y;
                if (code <= -2) ecum += w.Ecum[col_off(-(code + 2), m, M, t.Pp) + p];
            }
            w.Eown[col_off(iu, m, M, t.Pp) + p] = eown;
            w.Ecum[col_off(iu, m, M, t.Pp) + p] = ecum;
        }
        if (tile + 1 < t1) {
            s0 = n0;
            s1 = n1;
            if (one) load_msg8(a0, t, w, m, M, d0, p + kTileP, g, s0);
            if (two) load_msg8(a1, t, w, m, M, d1, p + kTileP, g, s1);
            if (tile + 2 < t1) { n0 = child_state(t, d0, p + 2 * kTileP); n1 = child_state(t, d1, p + 2 * kTileP); }
        }
        __syncthreads();
        // message to the parent: (P_u D_u)_i = sum_j P[i][j] D_j
        if (!root) tile_mm_store(f, sD, w.Ms + part_off(iu, m, M, t.Pp) + size_t(tile) * kTileP, Pp);
    }
}

// --------------------------------------------------------------------- root
__global__ void k_root(Topo t, Model md, Work w) {
    const int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= t.Pp) return;
    const int ir = t.iidx[t.root], M = md.M;
    const double wt = t.w[p];
    pdl_enter();
    double L[kMaxRateClasses], ll[kMaxRateClasses];
    for (int m = 0; m < M; ++m) {
        const double* D = w.D + part_off(ir, m, M, t.Pp) + p;
        double s = 0.0;
        if (t.S > kFewStates) {
            for (int i = 0; i < SP; ++i) s = fma(md.pi[i], D[size_t(i) * t.Pp], s);
        } else {                                   // h3g_few.cu leaves the other rows unwritten
            for (int i = 0; i < kFewStates; ++i) s = fma(md.pi[i], D[size_t(i) * t.Pp], s);
        }
        L[m] = s;
        ll[m] = s > 0.0 ? log(s) - double(w.Ecum[col_off(ir, m, M, t.Pp) + p]) * 0.69314718055994530942 : -1e20;
    }
    double site = -1e20, contrib = 0.0;
    bool ok = false;
    if (M == 1) {
        if (L[0] > 0.0) {
            ok = true; site = ll[0]; contrib = wt * ll[0];
            w.f[p] = wt / L[0];
        } else {
            w.f[p] = 0.0;
        }
        w.rw[p] = 0.0;
    } else {
        double mx = -INFINITY;
        for (int m = 0; m < M; ++m)
            if (md.rate_w[m] > 1e-12 && L[m] > 0.0) mx = fmax(mx, log(md.rate_w[m]) + ll[m]);
        double post[kMaxRateClasses], se = 0.0;
        for (int m = 0; m < M; ++m) {
            post[m] = 0.0;
            if (mx > -1e19 && md.rate_w[m] > 1e-12 && L[m] > 0.0) { post[m] = exp(log(md.rate_w[m]) + ll[m] - mx); se += post[m]; }
        }
        if (mx > -1e19 && se > 0.0) { ok = true; site = mx + log(se); contrib = wt * site; }
        for (int m = 0; m < M; ++m) {
            const double pw = ok ? post[m] / se : 0.0;
            w.f[size_t(m) * t.Pp + p] = (ok && pw > 1e-12) ? wt * pw / L[m] : 0.0;
            w.rw[size_t(m) * t.Pp + p] = ok ? wt * pw / md.rate_w[m] : 0.0;
        }
    }
    if (!ok && md.sentinel) contrib = wt * -1e20;
    w.contrib[p] = contrib;
    w.site[p] = site;
}

// ------------------------------------------------------------------ outside
// The outside partials of the internal children of one depth's nodes: with u the parent of c,
// V_c = 2^{e_u} U_u o prod_{s != c} (P_s D_s), U_c = P_c^T V_c, and f V_c for the gradient.  grid and tiles as
// k_inside, `kids` the children.  Leaves have no outside partial, and their V is formed where the gradient uses
// it (k_accumA_leaf): storing it for them was half of this kernel's CTAs and the gradient's largest stream
// (1024 taxa x 1200 codons x 4 rates: 4.87 -> 2.81 ms).
__global__ void __launch_bounds__(256, 2) k_outside(Topo t, Model md, Work w, const int* __restrict__ kids, int tiles) {
    __shared__ __align__(16) double sV[SP * kDL];
    __shared__ double smax[kGroups * kTileP];
    const int c = kids[blockIdx.y], m = blockIdx.z, g = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int u = t.parent[c], iu = t.iidx[u], ic = t.iidx[c], M = md.M;
    const int k0 = t.ch_off[u], k1 = t.ch_off[u + 1];
    const size_t Pp = size_t(t.Pp);
    const bool at_root = u == t.root;
    const int ks = t.kdesc[k0].x == c ? k0 + 1 : k0;              // the first sibling
    const bool sib = ks < k1, more = k1 - k0 > 2;
    const int2 ds = sib ? t.kdesc[ks] : make_int2(0, -1);
    const int* eo = w.Eown + col_off(iu, m, M, t.Pp);
    const double* fp = w.f + size_t(m) * Pp;
    const int t0 = blockIdx.x * tiles, t1 = min(t0 + tiles, t.Pp / kTileP);
    const size_t oc = part_off(ic, m, M, t.Pp), ou = part_off(at_root ? ic : iu, m, M, t.Pp);
    auto load_u = [&](double (&a)[8], int p) {
        const double* src = w.U + ou + size_t(8 * g) * Pp + p;
#pragma unroll
        for (int q = 0; q < 8; ++q) a[q] = at_root ? md.pi[8 * g + q] : src[q * Pp];
    };
    double a[8], b[8];
    int p = t0 * kTileP + lane;
    int st = child_state(t, ds, p), nx = 0;
    pdl_enter();                                                  // above: the problem's tables and patterns only
    int e = eo[p];
    double f = fp[p];
    load_u(a, p);
    if (sib) load_msg8(b, t, w, m, M, ds, p, g, st);
    const RowFrags fr = load_rows(w.PT + mat_off(m, c, t.n));
    if (t0 + 1 < t1) nx = child_state(t, ds, p + kTileP);
    for (int tile = t0; tile < t1; ++tile, p += kTileP) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = sib ? a[q] * b[q] : a[q];
        int ev = e - renorm_if_small(v, smax, g, lane, t.S);      // (its barrier: the last tile's products are done with sV)
        if (more)
            for (int k = ks + 1; k < k1; ++k) {
                const int2 d = t.kdesc[k];
                if (d.x == c) continue;
                double x[8];
                load_msg8(x, t, w, m, M, d, p, g, child_state(t, d, p));
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] *= x[q];
                ev -= renorm_if_small(v, smax, g, lane, t.S);
            }
        if (ev != 0) {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = ldexp(v[q], ev);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) sV[(8 * g + q) * kDL + lane] = v[q];
        double* vf = w.Vf + oc + size_t(8 * g) * Pp + p;
#pragma unroll
        for (int q = 0; q < 8; ++q) vf[q * Pp] = f * v[q];
        if (tile + 1 < t1) {
            st = nx;
            load_u(a, p + kTileP);
            if (sib) load_msg8(b, t, w, m, M, ds, p + kTileP, g, st);
            e = eo[p + kTileP];
            f = fp[p + kTileP];
            if (tile + 2 < t1) nx = child_state(t, ds, p + 2 * kTileP);
        }
        __syncthreads();
        tile_mm_store(fr, sV, w.U + oc + size_t(tile) * kTileP, Pp);       // (U_c)_i = sum_j PT[i][j] V_j
    }
}

// ------------------------------------------------------------------ accum A
// A_{m,b,chunk} = sum_{p in chunk} f V_b[:, p] D_b[:, p]^T.
//
// Internal branches on the FP64 tensor cores: C = X Y^T with X = f V (64 states x patterns), Y = D, K = the pattern
// axis.  8 warps as mm64 (warp w: rows 16(w/2) .. +16, columns 32(w%2) .. +32, 2 x 4 tiles of 8x8), 32 patterns
// per stage, stages double-buffered by 16-byte cp.async.  grid (branches, M, nchunk), block 256.
constexpr int kAccP = 32;                                      // patterns per stage
constexpr int kAL = kAccP + 4;                                 // row stride of a staged tile (doubles)
constexpr size_t kAccStage = size_t(2) * SP * kAL;             // V and D tiles of one stage
static const size_t kAccIntSmem = 2 * kAccStage * sizeof(double);

__device__ __forceinline__ void accumA_int(double* smA, const Topo& t, const Model& md, const Work& w, int b) {
    const int m = blockIdx.y, ck = blockIdx.z, tid = threadIdx.x, M = md.M;
    const size_t Pp = size_t(t.Pp);
    const int p_begin = ck * w.chunk, nst = (min(t.Pp, p_begin + w.chunk) - p_begin) / kAccP;
    const size_t o = part_off(t.iidx[b], m, M, t.Pp) + p_begin;
    // 64 state rows x 32 patterns of Vf and D into buffer st & 1
    auto stage = [&](int st) {
        double* sV = smA + size_t(st & 1) * kAccStage;
        double* sD = sV + SP * kAL;
        const size_t os = o + size_t(st) * kAccP;
#pragma unroll
        for (int i = 0; i < SP * (kAccP / 2) / 256; ++i) {
            const int c = tid + 256 * i, r = c / (kAccP / 2), q2 = c % (kAccP / 2);
            cp_async16_f64(sV + r * kAL + 2 * q2, w.Vf + os + size_t(r) * Pp + 2 * q2);
            cp_async16_f64(sD + r * kAL + 2 * q2, w.D + os + size_t(r) * Pp + 2 * q2);
        }
        asm volatile("cp.async.commit_group;" ::: "memory");
    };
    const int lane = tid & 31, wp = tid >> 5, g = lane >> 2, q = lane & 3;
    const int r0 = 16 * (wp >> 1), c0 = 32 * (wp & 1);
    Frag64 acc;
    frag_zero(acc);
    pdl_enter();                                 // above: the problem's tables only
    stage(0);
    for (int st = 0; st < nst; ++st) {
        if (st + 1 < nst) stage(st + 1);
        else asm volatile("cp.async.commit_group;" ::: "memory");
        asm volatile("cp.async.wait_group 1;" ::: "memory");
        __syncthreads();
        const double* sV = smA + size_t(st & 1) * kAccStage;
        const double* sD = sV + SP * kAL;
#pragma unroll
        for (int k = 0; k < kAccP; k += 4) {
            double x[2], y[4];
#pragma unroll
            for (int i = 0; i < 2; ++i) x[i] = sV[(r0 + 8 * i + g) * kAL + k + q];
#pragma unroll
            for (int j = 0; j < 4; ++j) y[j] = sD[(c0 + 8 * j + g) * kAL + k + q];
#pragma unroll
            for (int i = 0; i < 2; ++i)
#pragma unroll
                for (int j = 0; j < 4; ++j) dmma(acc.v[i][j][0], acc.v[i][j][1], x[i], y[j]);
        }
        __syncthreads();                         // the buffer is refilled by the next iteration's stage
    }
    double* dst = w.Apart + ((size_t(b) * M + m) * w.nchunk + ck) * SP2;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<double2*>(dst + frag_row(i) * SP + frag_col(j, 0)) = make_double2(acc.v[i][j][0], acc.v[i][j][1]);
}

__global__ void __launch_bounds__(256) k_accumA_int(Topo t, Model md, Work w, const int* __restrict__ branches) {
    extern __shared__ __align__(16) double smA[];
    accumA_int(smA, t, md, w, branches[blockIdx.x]);
}

// Leaf branches: D is a 0/1 vector, one state of each pattern for an unambiguous codon, so A[:, s] is the sum of the f V
// columns of the patterns in state s: 64 additions a pattern instead of a 64 x 64 outer product.  `leaves` holds
// one leaf, or the two of a node whose children are just these (x, y; y = -1 without): V of both comes from one read
// of U and the two messages.  Warp w owns the columns j with j % 8 = w (shared memory [column][64 rows], two rows a
// lane), walks the stage's patterns in those states in pattern order (a fixed order), and adds a pattern known only up
// to a set of codons to each of the set's columns; patterns without information (every state) are summed
// apart, pattern % 8 = w, and added to every column at the end.  grid (entries, M, nchunk), block 256.
// 1.60 ms for the 1024 leaves of the tree above; as outer products of a stored f V (1.32 ms), the kernel that stored it
// took 2 ms more.  Tried: each leaf alone with its rows of P^T fetched ahead (1.92 ms), V formed in this layout (2.40 ms).
constexpr int kLV = kAccP + 1;                                 // row stride of a V tile: a column's rows in 16 banks
constexpr int kLA = SP + 1;                                    // row stride of a column of A
constexpr int kLCols = SP + kGroups;
static const size_t kAccLeafSmem = (2 * SP * kLV + 2 * kLCols * kLA + kGroups * kTileP) * sizeof(double);

// the stage's V tile (sV; own: the observed state at the lane's pattern p) added to the columns of a leaf's A
__device__ __forceinline__ void leaf_add(double* sA, const double* sV, int own, const uint64_t* masks, int p, uint64_t all_mask, int g, int lane) {
    auto add = [&](int col, int x) {
        double* c = sA + col * kLA + lane;
        const double v0 = sV[lane * kLV + x], v1 = sV[(lane + 32) * kLV + x], c0 = c[0], c1 = c[32];
        c[0] = c0 + v0;
        c[32] = c1 + v1;
    };
    for (unsigned hit = __ballot_sync(0xffffffffu, own >= 0 && (own & 7) == g); hit; hit &= hit - 1) {
        const int x = __ffs(int(hit)) - 1;
        add(__shfl_sync(0xffffffffu, own, x), x);
    }
    unsigned rest = __ballot_sync(0xffffffffu, own < 0);
    if (rest) {
        uint64_t mk = own >= 0 || !masks ? 0 : masks[p];
        mk = mk == 0 || (mk & all_mask) == all_mask ? ~uint64_t(0) : mk & all_mask;     // ~0: no information
        for (; rest; rest &= rest - 1) {
            const int x = __ffs(int(rest)) - 1;
            uint64_t set = __shfl_sync(0xffffffffu, mk, x);
            if (set == ~uint64_t(0)) {
                if ((x & 7) == g) add(SP + g, x);
                continue;
            }
            for (set &= 0x0101010101010101ull << g; set; set &= set - 1) add(__ffsll((long long)set) - 1, x);
        }
    }
}

// kMany: the leaves of nodes with more than kFewKids children, alone.  Their time is the chain of siblings, so the
// siblings' descriptors, states and messages are loaded three, two and one ahead.  A star of 100 leaves x 3000 patterns
// takes 4.72 ms in place of 6.85 (with V stored: the outside pass 5.04, this 0.12), of 50 x 1000 459 us in place of
// 636 (451 and 34), of 12 x 100 31 us in place of 39.  With up to 9 children it is no faster (ladder of 9-child nodes: 108 us
// each way), and its registers would cost the pairs a third (256 taxa x 2000 codons 547 us in place of 407).
template <bool kMany>
__device__ __forceinline__ void accumA_leaf(double* smA, const Topo& t, const Model& md, const Work& w, int2 cc) {
    double* sA = smA + 2 * SP * kLV;
    double* smax = sA + 2 * kLCols * kLA;
    const int m = blockIdx.y, ck = blockIdx.z, tid = threadIdx.x, M = md.M;
    const int g = tid >> 5, lane = tid & 31;
    const bool pair = !kMany && cc.y >= 0;
    const int u = t.parent[cc.x], iu = t.iidx[u], k0 = t.ch_off[u], k1 = t.ch_off[u + 1];
    const size_t Pp = size_t(t.Pp);
    const bool at_root = u == t.root;
    // the message of cc.x's first sibling (cc.y's, for a pair) and, for a pair, cc.x's own
    const int ks = t.kdesc[k0].x == cc.x ? k0 + 1 : k0;
    const bool sib = ks < k1, more = k1 - k0 > 2;
    const int2 ds = sib ? t.kdesc[ks] : make_int2(0, -1), dx = make_int2(cc.x, t.taxon[cc.x]);
    const int tx = dx.y, ty = pair ? ds.y : -1;
    const int p_begin = ck * w.chunk, nst = (min(t.Pp, p_begin + w.chunk) - p_begin) / kAccP;
    const int* eo = w.Eown + col_off(iu, m, M, t.Pp);
    const double* fp = w.f + size_t(m) * Pp;
    const size_t ou = part_off(iu, m, M, t.Pp);
    auto load_u = [&](double (&a)[8], int p) {
        const double* src = w.U + ou + size_t(8 * g) * Pp + p;
#pragma unroll
        for (int q = 0; q < 8; ++q) a[q] = at_root ? md.pi[8 * g + q] : src[q * Pp];
    };
    for (int x = tid; x < (pair ? 2 : 1) * kLCols * kLA; x += 256) sA[x] = 0.0;
    double a[8], b[8], bx[8];
    int p = p_begin + lane;
    int own_x = child_state(t, dx, p), own_s = child_state(t, ds, p);
    pdl_enter();                                                  // above: the problem's tables and patterns only
    int e = eo[p];
    double f = fp[p];
    load_u(a, p);
    if (sib) load_msg8(b, t, w, m, M, ds, p, g, own_s);
    if (pair) load_msg8(bx, t, w, m, M, dx, p, g, own_x);
    int next_x = 0, next_s = 0;
    if (nst > 1) { next_x = child_state(t, dx, p + kAccP); next_s = child_state(t, ds, p + kAccP); }
    for (int st = 0; st < nst; ++st, p += kAccP) {
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = sib ? a[q] * b[q] : a[q];
        int ev = e - renorm_if_small(v, smax, g, lane, t.S);      // (its barrier: the last stage's additions are done with sV)
        if constexpr (kMany) {
            auto desc = [&](int k) { return k < k1 ? t.kdesc[k] : make_int2(cc.x, -1); };
            int2 d0 = desc(ks + 1), d1 = desc(ks + 2), d2 = desc(ks + 3);
            int s1 = child_state(t, d1, p);
            double x[8];
            load_msg8(x, t, w, m, M, d0, p, g, child_state(t, d0, p));
            for (int k = ks + 1; k < k1; ++k) {
                const int2 d3 = desc(k + 3);
                const int s2 = child_state(t, d2, p);
                double next[8];
                if (k + 1 < k1) load_msg8(next, t, w, m, M, d1, p, g, s1);
                if (d0.x != cc.x) {
#pragma unroll
                    for (int q = 0; q < 8; ++q) v[q] *= x[q];
                    ev -= renorm_if_small(v, smax, g, lane, t.S);
                }
#pragma unroll
                for (int q = 0; q < 8; ++q) x[q] = next[q];
                d0 = d1; d1 = d2; d2 = d3; s1 = s2;
            }
        } else if (more) {
            for (int k = ks + 1; k < k1; ++k) {
                const int2 d = t.kdesc[k];
                if (d.x == cc.x) continue;
                double x[8];
                load_msg8(x, t, w, m, M, d, p, g, child_state(t, d, p));
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] *= x[q];
                ev -= renorm_if_small(v, smax, g, lane, t.S);
            }
        }
        if (ev != 0) {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = ldexp(v[q], ev);
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) smA[(8 * g + q) * kLV + lane] = f * v[q];
        if (pair) {
#pragma unroll
            for (int q = 0; q < 8; ++q) v[q] = a[q] * bx[q];
            const int ey = e - renorm_if_small(v, smax, g, lane, t.S);
            if (ey != 0) {
#pragma unroll
                for (int q = 0; q < 8; ++q) v[q] = ldexp(v[q], ey);
            }
#pragma unroll
            for (int q = 0; q < 8; ++q) smA[(SP + 8 * g + q) * kLV + lane] = f * v[q];
        }
        const int sx = own_x, sy = own_s;
        if (st + 1 < nst) {
            own_x = next_x;
            own_s = next_s;
            load_u(a, p + kAccP);
            if (sib) load_msg8(b, t, w, m, M, ds, p + kAccP, g, own_s);
            if (pair) load_msg8(bx, t, w, m, M, dx, p + kAccP, g, own_x);
            e = eo[p + kAccP];
            f = fp[p + kAccP];
            if (st + 2 < nst) { next_x = child_state(t, dx, p + 2 * kAccP); next_s = child_state(t, ds, p + 2 * kAccP); }
        }
        __syncthreads();
        leaf_add(sA, smA, sx, tx < 0 ? nullptr : t.masks + size_t(tx) * Pp, p, t.all_mask, g, lane);
        if (pair) leaf_add(sA + kLCols * kLA, smA + SP * kLV, sy, ty < 0 ? nullptr : t.masks + size_t(ty) * Pp, p, t.all_mask, g, lane);
    }
    __syncthreads();
    for (int k = 0; k < (pair ? 2 : 1); ++k) {
        const double* A = sA + k * kLCols * kLA;
        double* dst = w.Apart + ((size_t(k ? cc.y : cc.x) * M + m) * w.nchunk + ck) * SP2;
        for (int x = tid; x < SP2; x += 256) {
            const int i = x >> 6, j = x & 63;
            double every = 0.0;
#pragma unroll
            for (int q = 0; q < kGroups; ++q) every += A[(SP + q) * kLA + i];
            dst[x] = j < t.S ? A[j * kLA + i] + every : 0.0;
        }
    }
}

template <bool kMany>
__global__ void __launch_bounds__(256, 2) k_accumA_leaf(Topo t, Model md, Work w, const int2* __restrict__ leaves) {
    extern __shared__ __align__(16) double smA[];
    accumA_leaf<kMany>(smA, t, md, w, leaves[blockIdx.x]);
}

// Both where they fit side by side (kAccSideBySide CTAs): a checkpoint block's few branches or a small gene leave most SMs
// idle, and two launches wait for each other.  256 taxa x 2000 codons x 2 rates in 33 blocks 14.2 -> 11.6 ms an
// evaluation, 600 x 1000 in 6 blocks 3.54 -> 3.20, in 80 17.5 -> 15.0; a star of 12 x 60 80 -> 70 us.
// The leaves come first: theirs is the longer chain.  grid (n_leaves + internal branches, M, nchunk), block 256.
__global__ void __launch_bounds__(256, 2) k_accumA_both(Topo t, Model md, Work w, const int2* __restrict__ leaves, int n_leaves,
                                                        const int* __restrict__ branches) {
    extern __shared__ __align__(16) double smA[];
    const int x = blockIdx.x;
    if (x < n_leaves) accumA_leaf<false>(smA, t, md, w, leaves[x]);
    else accumA_int(smA, t, md, w, branches[x - n_leaves]);
}
constexpr long kAccSideBySide = 2 * 148;

__device__ __forceinline__ double block_sum_256(double x, double* red) {
    for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
    const int lane = threadIdx.x & 31, wid = threadIdx.x >> 5;
    __syncthreads();
    if (lane == 0) red[wid] = x;
    __syncthreads();
    double s = 0.0;
    if (threadIdx.x == 0) for (int i = 0; i < 8; ++i) s += red[i];
    return s;   // valid on thread 0
}

// A_{m,b} = sum of the chunk partials in chunk order, and dlnL/dt_b's term
// <A_{m,b}, dP_{m,b}>.  grid (n, M), block 256.
__global__ void __launch_bounds__(256) k_areduce(Topo t, Model md, Work w) {
    pdl_enter();
    __shared__ double red[8];
    const int b = blockIdx.x, m = blockIdx.y, tid = threadIdx.x, n = t.n, M = md.M;
    if (b == t.root) return;
    const double* Ap = w.Apart + (size_t(b) * M + m) * w.nchunk * SP2 + tid;
    const double* dP = w.dP + mat_off(m, b, n) + tid;
    double* Af = w.Afull + (size_t(b) * M + m) * SP2 + tid;
    // a thread's 16 entries side by side: one entry after the other was 16 round trips to memory (19 us for the smallest genes)
    double s[SP2 / 256], d[SP2 / 256];
#pragma unroll
    for (int i = 0; i < SP2 / 256; ++i) { s[i] = Ap[256 * i]; d[i] = dP[256 * i]; }
    for (int ck = 1; ck < w.nchunk; ++ck)
#pragma unroll
        for (int i = 0; i < SP2 / 256; ++i) s[i] += Ap[size_t(ck) * SP2 + 256 * i];
    double g = 0.0;
#pragma unroll
    for (int i = 0; i < SP2 / 256; ++i) {
        Af[256 * i] = s[i];
        g = fma(s[i], d[i], g);
    }
    g = block_sum_256(g, red);
    if (tid == 0) w.gt[size_t(m) * n + b] = g;
}

// ------------------------------------------------------------------ frechet
// grid (G, M, nmod): CTA (g, m, k) walks the branches b = g, g+G, ... that use
// model k (test branches for k < K, background branches for k = K), computes
// the spectral transform At = U_k^T A_{m,b} V_k^T (two FP64 tensor-core products,
// mm64) and accumulates H += c_k At o E(lambda, tau_b) in registers
// (likelihood.hpp:1428-1471), plus the diagonal sums for d/dc_k and the d mu term.
// block 256, dynamic smem 3 x 64 x LDM doubles (U_k^T, V_k^T, A then T).
__global__ void __launch_bounds__(256) k_frechet(Topo t, Model md, Work w, int G) {
    pdl_enter();
    extern __shared__ __align__(16) double sm[];
    double* sUT = sm;                     // U_k^T: sUT[r][l] = U[l][r]
    double* sVT = sm + SP * LDM;          // V_k^T: sVT[l][c] = V[c][l]
    double* sA = sm + 2 * SP * LDM;       // A_{m,b}, then T = U^T A
    __shared__ double se[SP];
    __shared__ double red[8];
    const int g = blockIdx.x, m = blockIdx.y, k = blockIdx.z, tid = threadIdx.x, n = t.n, M = md.M;
    for (int e = tid; e < SP2; e += 256) {
        const int x = e >> 6, y = e & 63;                 // coalesced reads of U[x][y], V[x][y]
        sUT[y * LDM + x] = md.U[size_t(k) * SP2 + e];
        sVT[y * LDM + x] = md.V[size_t(k) * SP2 + e];
    }
    const double* lam = md.lam + size_t(k) * SP;
    Frag64 H;
    frag_zero(H);
    double dg = 0.0, dq = 0.0;
    for (int b = g; b < n; b += G) {
        if (b == t.root) continue;
        const BranchModels bm = branch_models(md, b);
        if (k < bm.k0 || k >= bm.k1) continue;
        const double cw = class_weight(md, bm, k);
        const double tau = md.rates[m] * w.bl[b] * time_conv(md, k);
        __syncthreads();                                  // the previous branch is done with sA
        {
            const double* A = w.Afull + (size_t(b) * M + m) * SP2;
            for (int e = tid; e < SP2; e += 256) sA[(e >> 6) * LDM + (e & 63)] = __ldg(A + e);
        }
        if (tid < SP) se[tid] = exp(lam[tid] * tau);
        __syncthreads();
        Frag64 T;
        mm64(sUT, sA, T);                                 // T = U^T A
        __syncthreads();                                  // every warp is done with A: T overwrites it
#pragma unroll
        for (int i = 0; i < 2; ++i)
#pragma unroll
            for (int j = 0; j < 4; ++j)
                *reinterpret_cast<double2*>(sA + frag_row(i) * LDM + frag_col(j, 0)) = make_double2(T.v[i][j][0], T.v[i][j][1]);
        __syncthreads();
        Frag64 At;
        mm64(sA, sVT, At);                                // At = T V^T
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            const int r = frag_row(i);
            const double li = lam[r], ei = se[r];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int e = 0; e < 2; ++e) {
                    const int c = frag_col(j, e);
                    const double d = li - lam[c], ej = se[c], a = At.v[i][j][e];
                    const double E = fabs(d) < 1e-9 ? tau * ei : (ei - ej) / d;
                    H.v[i][j][e] = fma(cw * a, E, H.v[i][j][e]);
                    if (r == c) {
                        dg += ei * a;
                        dq += cw * tau * li * ei * a;
                    }
                }
        }
    }
    double* Hp = w.Hpart + ((size_t(k) * M + m) * G + g) * SP2;
#pragma unroll
    for (int i = 0; i < 2; ++i)
#pragma unroll
        for (int j = 0; j < 4; ++j)
            *reinterpret_cast<double2*>(Hp + frag_row(i) * SP + frag_col(j, 0)) = make_double2(H.v[i][j][0], H.v[i][j][1]);
    dg = block_sum_256(dg, red);
    dq = block_sum_256(dq, red);
    if (tid == 0) {
        const size_t o = (size_t(k) * M + m) * G + g;
        w.gc[o] = dg;
        w.stg[o] = dq;
    }
}

// H_k[e] = sum over (m, g) of the per-CTA partials (fixed order: four interleaved
// running sums, combined pairwise), then the directional contractions
// dirpart[x][k][block] = sum over this block's 256 entries of H_k o G_{x,k}.
// grid (nmod, 16), block 256.
__global__ void __launch_bounds__(256) k_hsum(Topo t, Model md, Work w, int G) {
    pdl_enter();
    __shared__ double red[8];
    const int k = blockIdx.x, e = blockIdx.y * 256 + threadIdx.x, M = md.M, nt = M * G;
    const double* hp = w.Hpart + size_t(k) * nt * SP2 + e;
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
    int i = 0;
    for (; i + 4 <= nt; i += 4) {
        s0 += hp[size_t(i) * SP2];
        s1 += hp[size_t(i + 1) * SP2];
        s2 += hp[size_t(i + 2) * SP2];
        s3 += hp[size_t(i + 3) * SP2];
    }
    for (; i < nt; ++i) s0 += hp[size_t(i) * SP2];
    const double h = (s0 + s1) + (s2 + s3);
    w.H[size_t(k) * SP2 + e] = h;
    for (int x = 0; x < md.ndirs; ++x) {
        const double v = block_sum_256(h * w.G[(size_t(x) * md.nmod + k) * SP2 + e], red);
        if (threadIdx.x == 0) w.dirpart[(size_t(x) * md.nmod + k) * 17 + blockIdx.y] = v;
    }
}

// G_{x,k} = V_k dQ_{x,k} U_k, rows [16rb, 16rb+16); block 0 also stores
// d mu = -sum_i pi_i dQ_ii.  Depends on the model only, so it runs on a side
// stream alongside the pruning passes.  grid (ndirs, nmod, 4), block 256,
// dynamic smem (64*64 + 16*64 + 16*64) doubles.
__global__ void __launch_bounds__(256) k_dir(Topo t, Model md, Work w) {
    pdl_enter();
    extern __shared__ __align__(16) double sm[];
    double* sX = sm;                 // dQ, later U_k
    double* sY = sm + SP2;           // (V dQ)[rows, :]
    double* sVr = sY + 16 * SP;      // V_k rows of the block
    __shared__ double red[8];
    const int x = blockIdx.x, k = blockIdx.y, rb = blockIdx.z, tid = threadIdx.x;
    const bool own = x >= md.ndirs_dense;                 // a per-model direction: model x - ndirs_dense only
    if (own && k != x - md.ndirs_dense) {
        double* Gz = w.G + (size_t(x) * md.nmod + k) * SP2 + size_t(16 * rb) * SP;
        for (int e = tid; e < 16 * SP; e += 256) Gz[e] = 0.0;
        if (rb == 0 && tid == 0) w.dirpart[(size_t(x) * md.nmod + k) * 17 + 16] = 0.0;
        return;
    }
    const double* dQ = own ? md.dQ + (size_t(md.ndirs_dense) * md.nmod + k) * SP2 : md.dQ + (size_t(x) * md.nmod + k) * SP2;
    stage_matrix(sX, dQ, tid, 256);
    for (int e = tid; e < 16 * SP; e += 256) sVr[e] = md.V[size_t(k) * SP2 + size_t(16 * rb) * SP + e];
    __syncthreads();
    const int r = tid >> 4, c0 = (tid & 15) * 4;   // 16 rows x 64 columns, 4 per thread
    double acc[4] = {0, 0, 0, 0};
    for (int l = 0; l < SP; ++l) {
        const double a = sVr[r * SP + l];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = fma(a, sX[l * SP + c0 + q], acc[q]);
    }
#pragma unroll
    for (int q = 0; q < 4; ++q) sY[r * SP + c0 + q] = acc[q];
    double dmu = 0.0;
    if (rb == 0 && tid < SP) dmu = -md.pi[tid] * dQ[tid * SP + tid];
    __syncthreads();
    stage_matrix(sX, md.U + size_t(k) * SP2, tid, 256);
    __syncthreads();
#pragma unroll
    for (int q = 0; q < 4; ++q) acc[q] = 0.0;
    for (int l = 0; l < SP; ++l) {
        const double a = sY[r * SP + l];
#pragma unroll
        for (int q = 0; q < 4; ++q) acc[q] = fma(a, sX[l * SP + c0 + q], acc[q]);
    }
    double* Gx = w.G + (size_t(x) * md.nmod + k) * SP2 + size_t(16 * rb + r) * SP + c0;
#pragma unroll
    for (int q = 0; q < 4; ++q) Gx[q] = acc[q];
    dmu = block_sum_256(dmu, red);
    if (rb == 0 && tid == 0) w.dirpart[(size_t(x) * md.nmod + k) * 17 + 16] = dmu;
}

// Fixed-order reductions of the small per-branch / per-pattern partials.
// One block of 256 threads.
__global__ void __launch_bounds__(256) k_small(Topo t, Model md, Work w, int grads) {
    pdl_enter();
    __shared__ double red[8];
    const int tid = threadIdx.x, n = t.n, M = md.M;
    // lnL: per-thread Neumaier over a strided slice, then a fixed tree
    double s = 0.0, c = 0.0;
    for (int p = tid; p < t.Pp; p += 256) {
        const double x = w.contrib[p], y = s + x;
        c += fabs(s) >= fabs(x) ? (s - y) + x : (x - y) + s;
        s = y;
    }
    double tot = block_sum_256(s + c, red);
    if (tid == 0) { w.out[0] = tot; w.out[1] = w.err ? double(*w.err) : 0.0; }
    if (!grads) return;
    for (int b = tid; b < n; b += 256) {
        double g = 0.0;
        if (b != t.root) for (int m = 0; m < M; ++m) g += w.gt[size_t(m) * n + b];
        w.out[2 + b] = g;
    }
    for (int k = 0; k < md.nmod; ++k) {
        double a = 0.0, z = 0.0;
        for (int idx = tid; idx < M * w.ngroups; idx += 256) {
            a += w.gc[size_t(k) * M * w.ngroups + idx];
            z += w.stg[size_t(k) * M * w.ngroups + idx];
        }
        a = block_sum_256(a, red);
        z = block_sum_256(z, red);
        if (tid == 0) {
            w.out[2 + n + k] = a;                 // d lnL / d (class or background weight of model k)
            w.out[2 + n + md.nmod + k] = z;
        }
    }
    for (int m = 0; m < M; ++m) {
        double a = 0.0;
        for (int p = tid; p < t.Pp; p += 256) a += w.rw[size_t(m) * t.Pp + p];
        a = block_sum_256(a, red);
        if (tid == 0) w.out[2 + n + 2 * md.nmod + m] = a;
    }
}

// ------------------------------------------------------------------ launch
static const size_t kDirSmem = (2 * SP2 + 16 * SP) * sizeof(double);
static const size_t kBuildSmem = size_t(2) * SP * LDM * sizeof(double);
static const size_t kFrechetSmem = size_t(3) * SP * LDM * sizeof(double);

void fp64_configure() {
    cudaFuncSetAttribute(k_build_P<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBuildSmem));
    cudaFuncSetAttribute(k_build_P<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kBuildSmem));
    cudaFuncSetAttribute(k_frechet, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kFrechetSmem));
    cudaFuncSetAttribute(k_dir, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kDirSmem));
    cudaFuncSetAttribute(k_accumA_int, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kAccIntSmem));
    cudaFuncSetAttribute(k_accumA_both, cudaFuncAttributeMaxDynamicSharedMemorySize, int(std::max(kAccIntSmem, kAccLeafSmem)));
    cudaFuncSetAttribute(k_accumA_leaf<false>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kAccLeafSmem));
    cudaFuncSetAttribute(k_accumA_leaf<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, int(kAccLeafSmem));
}

int launch_build_P(const Topo& t, const Model& md, const Work& w, cudaStream_t s) {
    launch_k(k_build_P<false>, dim3(t.n, md.M), 256, kBuildSmem, s, t, md, w, MixedWork{});
    return 1;
}
int launch_build_P_mixed(const Topo& t, const Model& md, const Work& w, const MixedWork& mw, cudaStream_t s) {
    launch_k(k_build_P<true>, dim3(t.n, md.M), 256, kBuildSmem, s, t, md, w, mw);
    return 1;
}
int launch_prep_given_P(const Topo& t, const Work& w, cudaStream_t s) {
    launch_k(k_prep_given_P, t.n, 256, 0, s, t, w);
    return 1;
}
// Tiles per CTA of the pruning kernels: one while the level leaves SMs without a CTA to spare, up to 8 (four waves of
// two CTAs per SM are left then, so an uneven last wave costs little).  In a batch the other slots fill those waves, so
// a launch keeps its share of them: 24 genes of 8 to 512 taxa in 8 slots, two evaluations, 44.0 -> 40.4 ms (twice the
// tiles 40.4, half the CTAs 42.3, twice the CTAs 41.6).
static int tiles_per_cta(int ntile, int nodes, int M, int share) {
    const long items = long(ntile) * nodes * M, ctas = std::max(148L, 4L * 2 * 148 / share);
    return int(std::max(1L, std::min({8L, long(ntile), items / ctas})));
}
int launch_inside_fp64(const Topo& t, const Model& md, const Work& w, const int* d_nodes, int count, cudaStream_t s) {
    const int nt = t.Pp / kTileP, k = tiles_per_cta(nt, count, md.M, w.share);
    launch_k(k_inside, dim3((nt + k - 1) / k, count, md.M), 256, 0, s, t, md, w, d_nodes, k);
    return 1;
}
int launch_root(const Topo& t, const Model& md, const Work& w, cudaStream_t s) {
    launch_k(k_root, (t.Pp + 127) / 128, 128, 0, s, t, md, w);
    return 1;
}
int launch_outside_fp64(const Topo& t, const Model& md, const Work& w, const int* d_kids, int count, cudaStream_t s) {
    const int nt = t.Pp / kTileP, k = tiles_per_cta(nt, count, md.M, w.share);
    launch_k(k_outside, dim3((nt + k - 1) / k, count, md.M), 256, 0, s, t, md, w, d_kids, k);
    return 1;
}
int launch_accumA_fp64(const Topo& t, const Model& md, const Work& w, const int* d_internal, int n_internal, const int2* d_leaves,
                       int n_leaves, int n_many, cudaStream_t s) {
    const bool both = n_internal && n_leaves && long(n_internal + n_leaves) * md.M * w.nchunk <= kAccSideBySide;
    if (both) {
        launch_k(k_accumA_both, dim3(n_leaves + n_internal, md.M, w.nchunk), 256, std::max(kAccIntSmem, kAccLeafSmem), s, t, md, w, d_leaves,
                 n_leaves, d_internal);
    } else {
        if (n_internal) launch_k(k_accumA_int, dim3(n_internal, md.M, w.nchunk), 256, kAccIntSmem, s, t, md, w, d_internal);
        if (n_leaves) launch_k(k_accumA_leaf<false>, dim3(n_leaves, md.M, w.nchunk), 256, kAccLeafSmem, s, t, md, w, d_leaves);
    }
    if (n_many) launch_k(k_accumA_leaf<true>, dim3(n_many, md.M, w.nchunk), 256, kAccLeafSmem, s, t, md, w, d_leaves + n_leaves);
    return both ? 1 + (n_many > 0) : (n_internal > 0) + (n_leaves > 0) + (n_many > 0);
}
int launch_frechet(const Topo& t, const Model& md, const Work& w, int want_global, cudaStream_t s) {
    launch_k(k_areduce, dim3(t.n, md.M), 256, 0, s, t, md, w);
    if (!want_global) return 1;
    launch_k(k_frechet, dim3(w.ngroups, md.M, md.nmod), 256, kFrechetSmem, s, t, md, w, w.ngroups);
    return 2;
}
int launch_global(const Topo& t, const Model& md, const Work& w, cudaStream_t s) {
    launch_k(k_hsum, dim3(md.nmod, SP2 / 256), 256, 0, s, t, md, w, w.ngroups);
    return 1;
}
int launch_dir(const Topo& t, const Model& md, const Work& w, cudaStream_t s) {
    if (md.ndirs <= 0) return 0;
    launch_k(k_dir, dim3(md.ndirs, md.nmod, 4), 256, kDirSmem, s, t, md, w);
    return 1;
}
// The evaluation's results as one FP64 vector on the device, in the order
// [lnl, grad_t (n, root 0), grad_dir (ndirs), grad_class_w (K), grad_rate_w (M), failed]:
// every entry is a sum over site patterns (grad_dir's d mu term multiplies one such sum by a
// model constant), so vectors of pattern shards add up to the whole alignment's.  The directional
// gradient is assembled here from the 16 Frechet partials per (direction, model) exactly as the
// host does for h3g_eval.  One block.
__global__ void k_pack_result(Topo t, Model md, Work w, int grads, int global, double* dst) {
    const int tid = threadIdx.x, n = t.n, K = md.K, M = md.M, nmod = md.nmod, ndirs = md.ndirs;
    const double* out = w.out;
    if (tid == 0) {
        dst[0] = out[0];
        dst[1 + n + ndirs + K + M] = out[1] != 0.0 ? 1.0 : 0.0;
    }
    for (int b = tid; b < n; b += blockDim.x) dst[1 + b] = (grads && b != t.root) ? out[2 + b] : 0.0;
    for (int x = tid; x < ndirs; x += blockDim.x) {
        double g = 0.0;
        if (global)
            for (int k = 0; k < nmod; ++k) {
                const double* d = w.dirpart + (size_t(x) * nmod + k) * 17;
                double v = 0.0;
                for (int q = 0; q < 16; ++q) v += d[q];
                if (md.time_mode == 1) v -= d[16] / fmax(md.mu[k], 1e-12) * out[2 + n + nmod + k];
                g += v;
            }
        dst[1 + n + x] = g;
    }
    for (int k = tid; k < K; k += blockDim.x) dst[1 + n + ndirs + k] = global ? out[2 + n + k] : 0.0;
    for (int m = tid; m < M; m += blockDim.x) dst[1 + n + ndirs + K + m] = grads ? out[2 + n + 2 * nmod + m] : 0.0;
}

int launch_pack_result(const Topo& t, const Model& md, const Work& w, int grads, int global, double* dst, cudaStream_t s) {
    launch_k(k_pack_result, 1, 256, 0, s, t, md, w, grads, global, dst);
    return 1;
}

int launch_small(const Topo& t, const Model& md, const Work& w, int grads, cudaStream_t s) {
    launch_k(k_small, 1, 256, 0, s, t, md, w, grads);
    return 1;
}

bool pdl_enabled() {
    static const bool on = [] { const char* e = std::getenv("H3G_NO_PDL"); return !(e && e[0] == '1'); }();
    return on;
}

}  // namespace h3g
