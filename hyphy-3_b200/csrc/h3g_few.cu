// h3g_few.cu — the FP64 pruning passes for models of at most four states (nucleotides).
//
// The 64-state passes pad such a model sixteen times over and launch one kernel per level.  Here one thread owns one
// pattern of one node, with its states in registers, and one CTA of 16 warps walks the whole tree for 32 patterns:
// patterns are independent, so a level waits for the one before it with a barrier of the CTA instead of a launch.
// What bounds a pass is that chain of levels: one warp's item in a narrow level (about 400 instructions and two trips to
// L2, 2 us).  Descriptors and observed states are therefore loaded two items and one item ahead, and an item's matrix
// beside its children's messages (behind them: 101 us instead of 85 us for the inside pass below).
// 256 taxa x 3000 nucleotide patterns, 41 levels: inside 85 us, outside 67 us, A 53 us; as 64-state passes 1148, 1291
// and 437 us.
//
//   k_inside_few    partials and messages, children before parents (likelihood.hpp:500-597)
//   k_outside_few   outside partials of internal nodes, parents before children (likelihood.hpp:612-761)
//   k_accumA_few    A_b = sum_p f V_b D_b^T, V formed from U and the siblings' messages
//
// Layouts, scale exponents and results are those of the 64-state passes (h3g_common.cuh), rows 4 .. 63 left out, so the
// root, the reductions and the rest of the evaluation are shared.
#include "h3g_few.cuh"
#include "h3g_kernels.h"

namespace h3g {

namespace {

// A child's message at pattern p (d: Topo::kdesc entry, st: its observed state if a leaf).
__device__ __forceinline__ void few_msg(double (&x)[kFewStates], const Topo& t, const Work& w, int m, int M, int2 d, int p, int st) {
    if (d.y <= -2) {
        const double* src = w.Ms + part_off(-(d.y + 2), m, M, t.Pp) + p;
#pragma unroll
        for (int q = 0; q < kFewStates; ++q) x[q] = src[size_t(q) * t.Pp];
        return;
    }
    const double* PTc = w.PT + mat_off(m, d.x, t.n);
    const double* src = PTc + st * SP;
    if (st < 0) {
        const uint64_t mk = d.y < 0 ? t.all_mask : t.masks[size_t(d.y) * t.Pp + p];
        if (mk == 0 || (mk & t.all_mask) == t.all_mask) {
            src = w.rs + (size_t(m) * t.n + d.x) * SP;
        } else {
#pragma unroll
            for (int q = 0; q < kFewStates; ++q) x[q] = 0.0;
#pragma unroll
            for (int j = 0; j < kFewStates; ++j)
                if ((mk >> j) & 1)
#pragma unroll
                    for (int q = 0; q < kFewStates; ++q) x[q] += PTc[j * SP + q];
            return;
        }
    }
    const double2 a = __ldg(reinterpret_cast<const double2*>(src)), b = __ldg(reinterpret_cast<const double2*>(src) + 1);
    x[0] = a.x; x[1] = a.y; x[2] = b.x; x[3] = b.y;
}

// v away from underflow by a power of two, as the 64-state passes scale a column; returns the shift applied
__device__ __forceinline__ int few_scale(double (&v)[kFewStates]) {
    double mx = 0.0;
#pragma unroll
    for (int q = 0; q < kFewStates; ++q) mx = fmax(mx, v[q]);
    if (mx <= 0.0 || mx >= 0x1p-256) return 0;
    const int sh = -ilogb(mx) - 1;
#pragma unroll
    for (int q = 0; q < kFewStates; ++q) v[q] = ldexp(v[q], sh);
    return sh;
}
// v *= x; returns the shift applied
__device__ __forceinline__ int few_mul(double (&v)[kFewStates], const double (&x)[kFewStates]) {
#pragma unroll
    for (int q = 0; q < kFewStates; ++q) v[q] *= x[q];
    return few_scale(v);
}

// The upper left corner of a padded 64 x 64 matrix (the same for the whole warp), and its product with x.  Loaded
// ahead of the messages: behind them it was a second trip to memory for every item.
struct FewMat { double2 r[2 * kFewStates]; };
__device__ __forceinline__ FewMat few_mat(const double* mat) {
    FewMat a;
#pragma unroll
    for (int i = 0; i < 2 * kFewStates; ++i) a.r[i] = __ldg(reinterpret_cast<const double2*>(mat + (i >> 1) * SP) + (i & 1));
    return a;
}
__device__ __forceinline__ void few_apply(double (&y)[kFewStates], const FewMat& a, const double (&x)[kFewStates]) {
#pragma unroll
    for (int i = 0; i < kFewStates; ++i) {
        const double2 p = a.r[2 * i], q = a.r[2 * i + 1];
        y[i] = fma(q.x, x[2], p.x * x[0]) + fma(q.y, x[3], p.y * x[1]);
    }
}

// grid (Pp / 32, M).  Items: {u, iidx[u], first child slot, end}, the first two children's kdesc.
__global__ void __launch_bounds__(32 * kFewWarps) k_inside_few(Topo t, Model md, Work w) {
    const int lane = threadIdx.x & 31, p = 32 * int(blockIdx.x) + lane, m = blockIdx.y, M = md.M;
    const size_t Pp = size_t(t.Pp);
    few_walk(
        t.few_in_lv, t.few_in_levels, t.few_in, threadIdx.x >> 5,
        [&](int4 d, int& s0, int& s1) { s0 = few_state(t, make_int2(d.x, d.y), p); s1 = few_state(t, make_int2(d.z, d.w), p); },
        [] { pdl_enter(); },
        [&](int4 a, int4 d, int s0, int s1) {
            const int u = a.x, iu = a.y, k0 = a.z, k1 = a.w;
            double v[kFewStates], x[kFewStates];
#pragma unroll
            for (int q = 0; q < kFewStates; ++q) v[q] = q < t.S ? 1.0 : 0.0;
            const FewMat pm = few_mat(w.P + mat_off(m, u, t.n));      // (the root's is not used)
            const int e0 = d.y <= -2 ? w.Ecum[col_off(-(d.y + 2), m, M, t.Pp) + p] : 0;
            const int e1 = d.w <= -2 ? w.Ecum[col_off(-(d.w + 2), m, M, t.Pp) + p] : 0;
            if (k0 < k1) few_msg(v, t, w, m, M, make_int2(d.x, d.y), p, s0);
            int eown = few_scale(v), ecum = e0 + e1;
            if (k0 + 1 < k1) {
                few_msg(x, t, w, m, M, make_int2(d.z, d.w), p, s1);
                eown += few_mul(v, x);
            }
            if (k0 + 2 < k1) {
                // a polytomy: descriptors three, states two and messages one child ahead.  One after the other they are a
                // chain of three loads for each child: a value of a star of 400 leaves x 32000 patterns took 1740 us (the
                // 64-state passes 1474), now 1052; of 100 leaves x 14400 257 (233), now 191
                auto desc = [&](int k) { return k < k1 ? t.kdesc[k] : make_int2(0, -1); };
                int2 c = desc(k0 + 2), c1 = desc(k0 + 3), c2 = desc(k0 + 4);
                int st1 = few_state(t, c1, p);
                few_msg(x, t, w, m, M, c, p, few_state(t, c, p));
                for (int k = k0 + 2; k < k1; ++k) {
                    const int2 c3 = desc(k + 3);
                    const int st2 = few_state(t, c2, p);
                    double next[kFewStates];
                    if (k + 1 < k1) few_msg(next, t, w, m, M, c1, p, st1);
                    if (c.y <= -2) ecum += w.Ecum[col_off(-(c.y + 2), m, M, t.Pp) + p];
                    eown += few_mul(v, x);
#pragma unroll
                    for (int q = 0; q < kFewStates; ++q) x[q] = next[q];
                    c = c1; c1 = c2; c2 = c3; st1 = st2;
                }
            }
            const size_t o = part_off(iu, m, M, t.Pp) + p, oc = col_off(iu, m, M, t.Pp) + p;
#pragma unroll
            for (int q = 0; q < kFewStates; ++q) w.D[o + q * Pp] = v[q];
            w.Eown[oc] = eown;
            w.Ecum[oc] = ecum + eown;
            if (u != t.root) {
                few_apply(x, pm, v);
#pragma unroll
                for (int q = 0; q < kFewStates; ++q) w.Ms[o + q * Pp] = x[q];
            }
        });
}

// V of branch c below u: 2^{e_u} U_u o the siblings' messages (x0: the first sibling's, if there is one)
__device__ __forceinline__ void few_outside(double (&v)[kFewStates], const Topo& t, const Model& md, const Work& w, int m, int M, int iu,
                                            bool at_root, int c, int2 ds, int ks, int k1, int st, int p) {
    const size_t Pp = size_t(t.Pp);
    const double* src = w.U + part_off(iu, m, M, t.Pp) + p;
    double x[kFewStates];
#pragma unroll
    for (int q = 0; q < kFewStates; ++q) v[q] = at_root ? md.pi[q] : src[q * Pp];
    int e = w.Eown[col_off(iu, m, M, t.Pp) + p];
    if (ks < k1) {
        few_msg(x, t, w, m, M, ds, p, st);
        e -= few_mul(v, x);
    }
    for (int k = ks + 1; k < k1; ++k) {
        const int2 d = t.kdesc[k];
        if (d.x == c) continue;
        few_msg(x, t, w, m, M, d, p, few_state(t, d, p));
        e -= few_mul(v, x);
    }
    if (e != 0)
#pragma unroll
        for (int q = 0; q < kFewStates; ++q) v[q] = ldexp(v[q], e);
}

// grid (Pp / 32, M).  Items, internal children: {c, iidx[parent], iidx[c], parent is the root}, {first sibling's kdesc,
// its slot, end of the parent's children}.
__global__ void __launch_bounds__(32 * kFewWarps) k_outside_few(Topo t, Model md, Work w) {
    const int lane = threadIdx.x & 31, p = 32 * int(blockIdx.x) + lane, m = blockIdx.y, M = md.M;
    const size_t Pp = size_t(t.Pp);
    few_walk(
        t.few_out_lv, t.few_out_levels, t.few_out, threadIdx.x >> 5,
        [&](int4 d, int& s0, int& s1) { s1 = 0; s0 = few_state(t, make_int2(d.x, d.y), p); },
        [] { pdl_enter(); },
        [&](int4 a, int4 d, int s0, int) {
            double v[kFewStates], x[kFewStates];
            const FewMat pm = few_mat(w.PT + mat_off(m, a.x, t.n));
            few_outside(v, t, md, w, m, M, a.y, a.w != 0, a.x, make_int2(d.x, d.y), d.z, d.w, s0, p);
            few_apply(x, pm, v);
            const size_t o = part_off(a.z, m, M, t.Pp) + p;
#pragma unroll
            for (int q = 0; q < kFewStates; ++q) w.U[o + q * Pp] = x[q];
        });
}

// grid (n, M, nchunk), block 256: a thread takes every 256th pattern of the chunk, then a fixed tree; the chunk's
// 64 x 64 partial is written whole, zero outside the corner.
__global__ void __launch_bounds__(256) k_accumA_few(Topo t, Model md, Work w) {
    constexpr int kE = kFewStates * kFewStates;
    __shared__ double red[8][kE];
    const int b = blockIdx.x, m = blockIdx.y, ck = blockIdx.z, tid = threadIdx.x, M = md.M;
    if (b == t.root) return;
    const int u = t.parent[b], iu = t.iidx[u], k0 = t.ch_off[u], k1 = t.ch_off[u + 1], ib = t.iidx[b];
    const int ks = t.kdesc[k0].x == b ? k0 + 1 : k0;
    const int2 ds = ks < k1 ? t.kdesc[ks] : make_int2(0, -1), db = make_int2(b, ib < 0 ? t.taxon[b] : -2);
    const size_t Pp = size_t(t.Pp);
    const int p_end = min(t.Pp, (ck + 1) * w.chunk);
    double acc[kE];
#pragma unroll
    for (int e = 0; e < kE; ++e) acc[e] = 0.0;
    pdl_enter();
    for (int p = ck * w.chunk + tid; p < p_end; p += 256) {
        double v[kFewStates], d[kFewStates];
        const int own = few_state(t, db, p);
        if (ib >= 0) {
            const double* src = w.D + part_off(ib, m, M, t.Pp) + p;
#pragma unroll
            for (int q = 0; q < kFewStates; ++q) d[q] = src[q * Pp];
        } else {
            const uint64_t mk = own >= 0 ? uint64_t(1) << own : (db.y < 0 ? 0 : t.masks[size_t(db.y) * Pp + p]);
            const bool any = own < 0 && (mk == 0 || (mk & t.all_mask) == t.all_mask);
#pragma unroll
            for (int q = 0; q < kFewStates; ++q) d[q] = q < t.S && (any || ((mk >> q) & 1)) ? 1.0 : 0.0;
        }
        few_outside(v, t, md, w, m, M, iu, u == t.root, b, ds, ks, k1, few_state(t, ds, p), p);
        const double f = w.f[size_t(m) * Pp + p];
#pragma unroll
        for (int i = 0; i < kFewStates; ++i) {
            v[i] *= f;
#pragma unroll
            for (int j = 0; j < kFewStates; ++j) acc[kFewStates * i + j] = fma(v[i], d[j], acc[kFewStates * i + j]);
        }
    }
#pragma unroll
    for (int e = 0; e < kE; ++e)
        for (int o = 16; o > 0; o >>= 1) acc[e] += __shfl_xor_sync(0xffffffffu, acc[e], o);
    if ((tid & 31) == 0)
#pragma unroll
        for (int e = 0; e < kE; ++e) red[tid >> 5][e] = acc[e];
    __syncthreads();
    double* dst = w.Apart + ((size_t(b) * M + m) * w.nchunk + ck) * SP2;
    for (int x = tid; x < SP2; x += 256) {
        const int i = x >> 6, j = x & 63;
        double s = 0.0;
        if (i < kFewStates && j < kFewStates)
            for (int q = 0; q < 8; ++q) s += red[q][kFewStates * i + j];
        dst[x] = s;
    }
}

}  // namespace

int launch_inside_few(const Topo& t, const Model& md, const Work& w, cudaStream_t s) {
    launch_k(k_inside_few, dim3(t.Pp / 32, md.M), 32 * kFewWarps, 0, s, t, md, w);
    return 1;
}
int launch_outside_few(const Topo& t, const Model& md, const Work& w, cudaStream_t s) {
    if (t.few_out_levels == 0) return 0;
    launch_k(k_outside_few, dim3(t.Pp / 32, md.M), 32 * kFewWarps, 0, s, t, md, w);
    return 1;
}
int launch_accumA_few(const Topo& t, const Model& md, const Work& w, cudaStream_t s) {
    launch_k(k_accumA_few, dim3(t.n, md.M, w.nchunk), 256, 0, s, t, md, w);
    return 1;
}

}  // namespace h3g
