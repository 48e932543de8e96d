// h3g_nuc.cu — the nucleotide GTR log-likelihood on the device (h3g_nuc_eval_from_P).
//
// LikelihoodEngine::compute_gtr_log_likelihood (likelihood.hpp:181-254) prunes every
// nucleotide pattern through the tree with 4 x 4 transition matrices.  Here one thread
// owns one pattern and walks the tree depth-first along an event list shared by all
// threads (open an internal node / close a node into its parent), so a warp reads the
// same transition matrix at every step (one broadcast) and there is no inter-thread
// dependency.  The partial of the node being accumulated stays in registers; opening an
// internal node parks its parent's partial in a [depth][pattern] buffer (consecutive
// threads, consecutive addresses), closing it brings the parent back.  Partials are
// rescaled by 2^256 when their maximum falls below 2^-256; L = pi . D_root, the site
// log-likelihood log L - E ln 2, or the reference's -1e20 when L <= 0; the weighted sum
// over patterns is a fixed-order Neumaier sum.  FP64 throughout.
//
// With fewer patterns than it takes to fill the GPU (kLevelBelow), the tree is walked
// level by level instead, partials stored per internal node: by one launch, in which a
// CTA of 16 warps takes 32 patterns through all levels (h3g_few.cuh), a warp per internal
// node of the level, or by a launch per level, a thread per node and pattern (walk_wins).
#include <algorithm>
#include <cmath>
#include <new>
#include <string>
#include <utility>
#include <vector>

#include "h3g_few.cuh"
#include "h3g_fel.h"

namespace h3g {

Topo problem_topo(h3g_problem* pr, int S);                // h3g_capi.cu
cudaStream_t problem_stream(h3g_problem* pr);
void*& problem_nuc_state(h3g_problem* pr);
int problem_max_state(h3g_problem* pr);
void problem_levels(h3g_problem* pr, const std::vector<int>** nodes, const std::vector<int>** off);

namespace {

constexpr int kNucT = 128;                                 // threads per block (patterns)
constexpr int kLvlT = 256;
// Nodes x patterns of a level below which a thread loads two children side by side: at its 96 registers two CTAs fit an SM, so
// that is one wave.  Above, one at a time and twice the CTAs: 256 taxa at random x 131000 patterns 824 us, in pairs 1239; below,
// a chain of 256 taxa x 16000 758 us, one at a time 1344.
constexpr size_t kPairBelow = size_t(148) * 2 * kLvlT;
constexpr int kSumT = 1024;
constexpr int kLevelBelow = 131072;                        // patterns: below, the level-by-level walk

struct NucState {
    int n_ev = 0, depth = 1, P = 0;
    size_t Pp = 0;
    int* d_ev = nullptr;
    double* d_P = nullptr;                                 // [n][16]
    double* d_pi = nullptr;                                // [4]
    double* d_site = nullptr;                              // [P]
    double4* d_stk = nullptr;                              // [depth][Pp]
    int* d_exp = nullptr;                                  // [depth][Pp]
    bool levels = false;                                   // level by level ...
    bool walk = false;                                     // ... in one launch
    double4* d_part = nullptr;                             // [NI][Pp]
    int* d_pexp = nullptr;                                 // [NI][Pp]
    double* d_lnl = nullptr;
    double* h_pin = nullptr;                               // lnl read back
    std::vector<void*> owned;
    ~NucState() {
        for (void* p : owned) cudaFree(p);
        if (h_pin) cudaFreeHost(h_pin);
    }
};

__global__ void __launch_bounds__(kNucT) k_nuc_lnl(Topo t, const int* __restrict__ ev, int n_ev, const double* __restrict__ P,
                                                    const double* __restrict__ pi, double4* __restrict__ stk,
                                                    int* __restrict__ sexp, double* __restrict__ site) {
    pdl_enter();
    const int p = int(blockIdx.x) * kNucT + int(threadIdx.x);
    if (p >= t.P) return;
    const size_t Pp = size_t(t.Pp);
    double d[4] = {1.0, 1.0, 1.0, 1.0};                     // partial of the innermost open node
    int E = 0, sp = -1;                                    // levels 0 .. sp - 1 are parked in stk
    for (int k = 0; k < n_ev; ++k) {
        const int code = __ldg(ev + k), node = code >> 1;
        if (code & 1) {                                    // open an internal node
            if (sp >= 0) {
                stk[size_t(sp) * Pp + p] = make_double4(d[0], d[1], d[2], d[3]);
                sexp[size_t(sp) * Pp + p] = E;
            }
            ++sp;
            d[0] = d[1] = d[2] = d[3] = 1.0;
            E = 0;
            continue;
        }
        double x[4];
        int Ex = 0;
        if (t.leaf[node]) {                                // likelihood.hpp:54-87
            const int tx = t.taxon[node];
            int st = -1;
            uint64_t mk = 0xF;
            if (tx >= 0) {
                st = t.states[size_t(tx) * Pp + p];
                if (!(st >= 0 && st < 4)) mk = t.masks[size_t(tx) * Pp + p];
            }
            if (st >= 0 && st < 4) {
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = i == st ? 1.0 : 0.0;
            } else if (mk == 0 || (mk & 0xF) == 0xF) {
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = 1.0;
            } else {
#pragma unroll
                for (int i = 0; i < 4; ++i) x[i] = ((mk >> i) & 1) ? 1.0 : 0.0;
            }
        } else {                                           // close an internal node: its partial is d
#pragma unroll
            for (int i = 0; i < 4; ++i) x[i] = d[i];
            Ex = E;
            --sp;
            const double4 v = stk[size_t(sp) * Pp + p];
            d[0] = v.x; d[1] = v.y; d[2] = v.z; d[3] = v.w;
            E = sexp[size_t(sp) * Pp + p];
        }
        const double* Pn = P + size_t(node) * 16;          // the same matrix for the whole warp
        double mx = 0.0;
#pragma unroll
        for (int i = 0; i < 4; ++i) {
            const double m = __ldg(Pn + 4 * i) * x[0] + __ldg(Pn + 4 * i + 1) * x[1] + __ldg(Pn + 4 * i + 2) * x[2] +
                             __ldg(Pn + 4 * i + 3) * x[3];
            d[i] *= m;
            mx = fmax(mx, d[i]);
        }
        E += Ex;
        if (mx > 0.0 && mx < 0x1p-256) {
#pragma unroll
            for (int i = 0; i < 4; ++i) d[i] *= 0x1p256;
            E += 256;
        }
    }
    const double L = pi[0] * d[0] + pi[1] * d[1] + pi[2] * d[2] + pi[3] * d[3];
    site[p] = L > 0.0 ? log(L) - double(E) * 0.69314718055994530942 : -1e20;
}

// A child at pattern p (c: Topo::kdesc entry, st: its observed state if a leaf): its matrix, partial and exponent.
struct NucChild { double2 P[8]; double x[4]; int E; };
__device__ __forceinline__ NucChild nuc_child(const Topo& t, const double* __restrict__ P, const double4* part, const int* pexp, int2 c,
                                              int st, int p) {
    NucChild o;
    const double2* Pn = reinterpret_cast<const double2*>(P + size_t(c.x) * 16);
#pragma unroll
    for (int i = 0; i < 8; ++i) o.P[i] = __ldg(Pn + i);
    o.E = 0;
    if (c.y <= -2) {
        const size_t at = size_t(-(c.y + 2)) * size_t(t.Pp) + p;
        const double4 v = part[at];
        o.x[0] = v.x; o.x[1] = v.y; o.x[2] = v.z; o.x[3] = v.w;
        o.E = pexp[at];
    } else {                                               // likelihood.hpp:54-87
        const uint64_t mk = st >= 0 ? uint64_t(1) << st : (c.y < 0 ? 0xF : t.masks[size_t(c.y) * size_t(t.Pp) + p]);
        const bool any = st < 0 && (mk == 0 || (mk & 0xF) == 0xF);
#pragma unroll
        for (int i = 0; i < 4; ++i) o.x[i] = any || ((mk >> i) & 1) ? 1.0 : 0.0;
    }
    return o;
}
__device__ __forceinline__ void nuc_take(double (&d)[4], int& E, const NucChild& c) {
    double mx = 0.0;
#pragma unroll
    for (int i = 0; i < 4; ++i) {
        const double2 a01 = c.P[2 * i], a23 = c.P[2 * i + 1];
        d[i] *= a01.x * c.x[0] + a01.y * c.x[1] + a23.x * c.x[2] + a23.y * c.x[3];
        mx = fmax(mx, d[i]);
    }
    E += c.E;
    if (mx > 0.0 && mx < 0x1p-256) {
#pragma unroll
        for (int i = 0; i < 4; ++i) d[i] *= 0x1p256;
        E += 256;
    }
}
// One internal node at one pattern: the product of its children's messages.  a, d4: its two few_in descriptors; s0, s1: the
// observed states of its first two children.
template <bool kPair>
__device__ __forceinline__ void nuc_node(const Topo& t, const double* __restrict__ P, const double* __restrict__ pi, double4* part,
                                         int* pexp, double* __restrict__ site, int4 a, int4 d4, int s0, int s1, int p) {
    const int k0 = a.z, k1 = a.w;
    double d[4] = {1.0, 1.0, 1.0, 1.0};
    int E = 0;
    if (kPair && k0 + 1 < k1) {                            // two side by side: one trip to memory
        const NucChild c0 = nuc_child(t, P, part, pexp, make_int2(d4.x, d4.y), s0, p);
        const NucChild c1 = nuc_child(t, P, part, pexp, make_int2(d4.z, d4.w), s1, p);
        nuc_take(d, E, c0);
        nuc_take(d, E, c1);
    } else if (k0 < k1) {
        nuc_take(d, E, nuc_child(t, P, part, pexp, make_int2(d4.x, d4.y), s0, p));
    }
    if (!kPair && k0 + 1 < k1) nuc_take(d, E, nuc_child(t, P, part, pexp, make_int2(d4.z, d4.w), s1, p));
    for (int k = k0 + 2; k < k1; ++k) {
        const int2 c = t.kdesc[k];
        nuc_take(d, E, nuc_child(t, P, part, pexp, c, few_state(t, c, p), p));
    }
    if (a.x == t.root) {
        if (p >= t.P) return;
        const double L = pi[0] * d[0] + pi[1] * d[1] + pi[2] * d[2] + pi[3] * d[3];
        site[p] = L > 0.0 ? log(L) - double(E) * 0.69314718055994530942 : -1e20;
    } else {
        const size_t o = size_t(a.y) * size_t(t.Pp) + p;
        part[o] = make_double4(d[0], d[1], d[2], d[3]);
        pexp[o] = E;
    }
}

// The whole tree, level by level; grid ceil(P / 32).
__global__ void __launch_bounds__(32 * kFewWarps) k_nuc_walk(Topo t, const double* __restrict__ P, const double* __restrict__ pi,
                                                             double4* part, int* pexp, double* __restrict__ site) {
    const int lane = threadIdx.x & 31, p = 32 * int(blockIdx.x) + lane;
    few_walk(
        t.few_in_lv, t.few_in_levels, t.few_in, threadIdx.x >> 5,
        [&](int4 d, int& s0, int& s1) { s0 = few_state(t, make_int2(d.x, d.y), p); s1 = few_state(t, make_int2(d.z, d.w), p); },
        [] { pdl_enter(); },
        [&](int4 a, int4 d, int s0, int s1) { nuc_node<true>(t, P, pi, part, pexp, site, a, d, s0, s1, p); });
}

// Nodes first .. first + cnt of one level, a thread per (node, pattern).
template <bool kPair>
__global__ void __launch_bounds__(kLvlT, kPair ? 1 : 4) k_nuc_level(Topo t, int first, int cnt, const double* __restrict__ P, const double* __restrict__ pi,
                                                     double4* part, int* pexp, double* __restrict__ site) {
    const size_t i = size_t(blockIdx.x) * kLvlT + threadIdx.x, P_ = size_t(t.P);
    if (i >= cnt * P_) return;
    const int node = first + int(i / P_), p = int(i % P_);
    const int4 a = t.few_in[2 * node], d = t.few_in[2 * node + 1];
    const int s0 = few_state(t, make_int2(d.x, d.y), p), s1 = few_state(t, make_int2(d.z, d.w), p);
    pdl_enter();                                           // the lower levels' partials are complete
    nuc_node<kPair>(t, P, pi, part, pexp, site, a, d, s0, s1, p);
}

// One block: weights x site log-likelihoods, Neumaier over every 1024th pattern, then a fixed tree of two-sums (the
// 1024 partial sums added up by one thread took 25 of this kernel's 27 us).
__device__ __forceinline__ void two_sum(double& s, double& c, double x, double xc) {
    const double t = s + x;
    c += xc + (fabs(s) >= fabs(x) ? (s - t) + x : (x - t) + s);
    s = t;
}
__global__ void __launch_bounds__(kSumT) k_nuc_sum(const double* __restrict__ site, const double* __restrict__ w, int P,
                                                   double* __restrict__ out) {
    pdl_enter();                                           // the site log-likelihoods are complete
    __shared__ double hi[kSumT / 32], lo[kSumT / 32];
    const int tid = threadIdx.x;
    double s = 0.0, c = 0.0;
    for (int i = tid; i < P; i += kSumT) two_sum(s, c, w[i] * site[i], 0.0);
    auto warp_sum = [&] {
        for (int o = 16; o > 0; o >>= 1) {
            const double x = __shfl_down_sync(0xffffffffu, s, o), xc = __shfl_down_sync(0xffffffffu, c, o);
            two_sum(s, c, x, xc);
        }
    };
    warp_sum();
    if ((tid & 31) == 0) { hi[tid >> 5] = s; lo[tid >> 5] = c; }
    __syncthreads();
    if (tid >= 32) return;
    s = hi[tid];
    c = lo[tid];
    warp_sum();
    if (tid == 0) *out = s + c;
}

// Whether the walk takes less time than a launch per level, by the time of each in microseconds.  The walk's CTAs have an
// SM to themselves (registers), so beyond 32 patterns an SM they run in waves, each as long as its chain of items: 1.25 a
// binary node, 0.75 each further child, every 16 nodes of a level one item; 28e-6 a node and pattern at least.  A launch per
// level costs 25 in all and for each level its launch and one node's chain, 2.9 and 0.65 each further child, or 22e-6
// a node and pattern if that is more.  Fits whole calls to 20 % where the two are far apart.  Walk / levels in us: a chain of
// 256 taxa x 16000 patterns 1397 / 759, x 64000 4728 / 871; a star of 100 x 8000 161 / 87, x 64000 764 / 102; 256 taxa at
// random x 16000 207 / 160, x 64000 610 / 440; 1024 taxa x 8000 306 / 281, x 64000 1795 / 1529.  (The walk is taken for the
// chain up to x 8000, 686; for the star at x 3000, 88; for the 256 taxa at x 8000, 117.)
bool walk_wins(const std::vector<int>& nodes, const std::vector<int>& off, const FelProblemView& v, int P, int sms) {
    const int waves = ((P + 31) / 32 + sms - 1) / sms;
    double chain = 0.0, levels = 25.0;
    for (size_t l = 0; l + 1 < off.size(); ++l) {
        const int width = off[l + 1] - off[l];
        int more = 0;
        for (int k = off[l]; k < off[l + 1]; ++k) more = std::max(more, v.ch_off[nodes[size_t(k)] + 1] - v.ch_off[nodes[size_t(k)]] - 2);
        chain += (width + kFewWarps - 1) / kFewWarps * (1.25 + 0.75 * more);
        levels += std::max(2.9 + 0.65 * more, 22e-6 * width * P);
    }
    return std::max(28e-6 * double(nodes.size()) * P, waves * chain) < levels;
}

// depth-first events (2 node + 1 opens an internal node, 2 node closes a node) and the
// largest number of internal nodes open at once
std::pair<std::vector<int>, int> dfs_events(const FelProblemView& v) {
    std::vector<int> ev;
    ev.reserve(2 * size_t(v.n));
    int open = 1, deepest = 1;
    std::vector<std::pair<int, int>> stk{{v.root, 0}};
    ev.push_back(2 * v.root + 1);
    while (!stk.empty()) {
        auto& [u, k] = stk.back();
        if (k < v.ch_off[u + 1] - v.ch_off[u]) {
            const int c = v.ch[v.ch_off[u] + k++];
            if (v.leaf[c]) {
                ev.push_back(2 * c);
            } else {
                ev.push_back(2 * c + 1);
                deepest = std::max(deepest, ++open);
                stk.push_back({c, 0});
            }
        } else {
            if (u != v.root) {
                ev.push_back(2 * u);
                --open;
            }
            stk.pop_back();
        }
    }
    return {ev, deepest};
}

NucState* nuc_state(h3g_problem* pr, const FelProblemView& v, std::string* err) {
    void*& slot = problem_nuc_state(pr);
    if (slot) return static_cast<NucState*>(slot);
    auto* s = new (std::nothrow) NucState;
    if (!s) { *err = "host allocation failed"; return nullptr; }
    const Topo t = problem_topo(pr, 4);
    auto [ev, deepest] = dfs_events(v);
    s->n_ev = int(ev.size());
    s->depth = deepest;
    s->P = t.P;
    s->Pp = size_t(t.Pp);
    s->levels = t.P < kLevelBelow;
    int sms = 148;
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, v.device);
    const std::vector<int>*nodes, *off;
    problem_levels(pr, &nodes, &off);
    s->walk = walk_wins(*nodes, *off, v, t.P, sms);
    auto take = [&](auto** p, size_t count) {
        void* q = nullptr;
        if (cudaMalloc(&q, std::max<size_t>(count, 1) * sizeof(**p)) != cudaSuccess) return false;
        s->owned.push_back(q);
        *p = static_cast<std::remove_reference_t<decltype(*p)>>(q);
        return true;
    };
    bool ok = take(&s->d_ev, ev.size()) && take(&s->d_P, size_t(v.n) * 16) && take(&s->d_pi, 4) &&
              take(&s->d_site, size_t(std::max(t.P, 1))) && take(&s->d_lnl, 1) &&
              cudaMallocHost(reinterpret_cast<void**>(&s->h_pin), sizeof(double)) == cudaSuccess &&
              cudaMemcpy(s->d_ev, ev.data(), ev.size() * sizeof(int), cudaMemcpyHostToDevice) == cudaSuccess;
    if (ok && s->levels)
        ok = take(&s->d_part, size_t(t.NI) * s->Pp) && take(&s->d_pexp, size_t(t.NI) * s->Pp);
    else if (ok)
        ok = take(&s->d_stk, size_t(deepest) * s->Pp) && take(&s->d_exp, size_t(deepest) * s->Pp);
    // the copies above come from pageable memory on the default stream, which the evaluator's
    // non-blocking stream does not wait for
    ok = ok && cudaStreamSynchronize(cudaStreamLegacy) == cudaSuccess;
    if (!ok) {
        *err = "device allocation failed";
        delete s;
        return nullptr;
    }
    slot = s;
    return s;
}

}  // namespace

void nuc_state_free(void* p) { delete static_cast<NucState*>(p); }

}  // namespace h3g

using namespace h3g;

extern "C" h3g_status h3g_nuc_eval_from_P(h3g_problem* pr, const double* P, const double* pi, double* lnl, double* site_lnl) {
    if (!pr) return H3G_ERR_ARG;
    FelProblemView v;
    if (!P || !pi || !lnl || !fel_problem_view(pr, &v)) { fel_set_error(pr, "h3g_nuc_eval_from_P: null argument"); return H3G_ERR_ARG; }
    if (problem_max_state(pr) >= 4) {
        fel_set_error(pr, "h3g_nuc_eval_from_P: the problem's patterns are not nucleotide patterns (a state is >= 4)");
        return H3G_ERR_ARG;
    }
    for (int i = 0; i < 4; ++i)
        if (!std::isfinite(pi[i]) || pi[i] < 0.0) { fel_set_error(pr, "h3g_nuc_eval_from_P: pi must be finite and >= 0"); return H3G_ERR_NUMERIC; }
    for (int b = 0; b < v.n; ++b)
        for (int e = 0; e < 16 && b != v.root; ++e)
            if (!std::isfinite(P[size_t(b) * 16 + e])) { fel_set_error(pr, "h3g_nuc_eval_from_P: non-finite transition matrix"); return H3G_ERR_NUMERIC; }
    std::string err;
    NucState* s = nuc_state(pr, v, &err);
    if (!s) { fel_set_error(pr, "h3g_nuc_eval_from_P: " + err); return H3G_ERR_OOM; }
    cudaStream_t st = problem_stream(pr);
    const Topo t = problem_topo(pr, 4);
    bool ok = cudaMemcpyAsync(s->d_P, P, size_t(v.n) * 16 * sizeof(double), cudaMemcpyHostToDevice, st) == cudaSuccess &&
              cudaMemcpyAsync(s->d_pi, pi, 4 * sizeof(double), cudaMemcpyHostToDevice, st) == cudaSuccess;
    if (ok && s->P > 0) {
        if (s->levels && !s->walk) {
            const std::vector<int>*nodes, *off;
            problem_levels(pr, &nodes, &off);
            for (size_t l = 0; l + 1 < off->size(); ++l) {
                const int first = (*off)[l], cnt = (*off)[l + 1] - first;
                if (cnt == 0) continue;
                const bool pair = size_t(cnt) * size_t(s->P) < kPairBelow;
                launch_k(pair ? k_nuc_level<true> : k_nuc_level<false>, int((size_t(cnt) * size_t(s->P) + kLvlT - 1) / kLvlT), kLvlT, 0, st, t, first, cnt,
                         static_cast<const double*>(s->d_P), static_cast<const double*>(s->d_pi), s->d_part, s->d_pexp, s->d_site);
            }
        } else if (s->levels) {
            launch_k(k_nuc_walk, (s->P + 31) / 32, 32 * kFewWarps, 0, st, t, static_cast<const double*>(s->d_P),
                     static_cast<const double*>(s->d_pi), s->d_part, s->d_pexp, s->d_site);
        } else {
            launch_k(k_nuc_lnl, (s->P + kNucT - 1) / kNucT, kNucT, 0, st, t, static_cast<const int*>(s->d_ev), s->n_ev,
                     static_cast<const double*>(s->d_P), static_cast<const double*>(s->d_pi), s->d_stk, s->d_exp, s->d_site);
        }
        launch_k(k_nuc_sum, 1, kSumT, 0, st, static_cast<const double*>(s->d_site), t.w, s->P, s->d_lnl);
    }
    ok = ok && cudaGetLastError() == cudaSuccess &&
         cudaMemcpyAsync(s->h_pin, s->d_lnl, sizeof(double), cudaMemcpyDeviceToHost, st) == cudaSuccess &&
         (!site_lnl || s->P == 0 ||
          cudaMemcpyAsync(site_lnl, s->d_site, size_t(s->P) * sizeof(double), cudaMemcpyDeviceToHost, st) == cudaSuccess) &&
         cudaStreamSynchronize(st) == cudaSuccess;
    if (!ok) { fel_set_error(pr, std::string("h3g_nuc_eval_from_P: ") + cudaGetErrorString(cudaGetLastError())); return H3G_ERR_CUDA; }
    *lnl = s->P > 0 ? *s->h_pin : 0.0;
    return H3G_OK;
}
