// h3g_jacobi.cuh — parallel cyclic Jacobi for a symmetric 64x64 FP64 matrix held in shared
// memory by one CTA: sweeps() for the per-site fits' eigensystems (h3g_fel.cu), whose searches compare
// likelihoods bit for bit, and for the main engine's FP64 models (h3g_eigen.cu); sweeps_sym(), on half of the
// matrix, for its mixed-precision models.
//
// Golub & Van Loan, "Matrix Computations" (Alg. 8.5.1 / 8.5.3): one sweep = 63 rounds of 32
// disjoint rotations (p_k, q_k), p < q, covering all 64 indices (circle schedule: seat k of round r
// pairs x = r + k with y = r - k mod 63, seat 0 pairs 63 with r).  A round replaces every 2x2 block
// (I, J) of A by R_I^T A_IJ R_J, the diagonal blocks by their exact annihilated values
// a_pp - t a_pq, a_qq + t a_pq and 0, and the columns of E by E R.  The sweeps stop when the
// off-diagonal mass is below 1e-30 of the total.
//
// One matrix is a chain of ~500 dependent rounds (8 sweeps), and shared-memory bandwidth is what a
// round costs once several matrices share an SM.  So:
//   - A warp of its own runs one round ahead: from the rotations of round r and the A before it, it forms
//     just the 32 entries that round r + 1 annihilates (one 2x2 block each, in the workers' arithmetic, so
//     with the same bits) and from them the rotations of round r + 1 (square root, divide, reciprocal
//     square root: the longest chain of a round), while the workers apply round r from one buffer into the
//     other: one barrier a round.
//   - A is stored by seat, not by index: x_k at position k, y_k at 32 + k.  From one round to the next the
//     occupants move to the neighbouring seat (x_k -> x_{k-1}, y_k -> y_{k+1}; y_0 <- x_1, x_31 <- y_31, 63
//     stays), so a worker stores its results one position on and all its addresses are fixed.  A row's 32 p
//     (or q) entries then lie in nearly as many banks whichever of x and y is the p, and no index is computed
//     modulo 63.
//   - E stays in the workers' registers, four threads to a row with eight seats each; a round passes two
//     entries per thread on through shared memory (E in shared memory cost as much bandwidth as A).
// A round takes 1540 cycles with one CTA on the SM and 1320 per matrix with two; it moves 1060 wavefronts through
// shared memory (A's loads and stores 750, the rest c, s and E's entries), which bounds the second figure.
// Measured, dense random 61-state matrices (8 sweeps) at 148 / 296 / 444 at once: 397 / 593 / 904 us; with A and E in
// shared memory by index and two barriers a round, the rotations between them: 874 / 1215 / 1695 us.  Tried: 512
// workers (437 / 679 / 1002), A and E on warps of their own (393 / 624 / 925), the rotation warp alone on
// its quarter of the SM (454 / 735 / 1068).
#pragma once

#include "h3g_common.cuh"

namespace h3g {
namespace jac {

constexpr int LD = SP + 1;                // row stride of the callers' A and E: column walks hit 16 distinct 8-byte banks
constexpr int kWorkers = 256;             // threads that update A and E
constexpr int kWarps = kWorkers / 32;
constexpr int kSeats = 8;                 // seats of E a worker holds
constexpr int kGroups = 32 / kSeats;      // workers that share a row of E
constexpr int kBlocks = 32 / kWarps;      // blocks of A a worker updates
constexpr int kThreads = kWorkers + 32;   // and the warp that computes the rotations
// A by position: rows 0 .. 31 hold x, 32 .. 63 y; columns 0 .. 31 x, 47 .. 78 y.  With y's columns one bank
// behind x's, the loads (x_k or y_k from lane k) and the stores one seat on (x_1 to y_0 and y_31 to x_31
// among them) hit 16 distinct banks per half warp but for the one where the roles change.
constexpr int kYCol = 47;
constexpr int kPitch = 80;
constexpr int kBuf = SP * kPitch;         // one buffer of A
constexpr size_t kSmem = size_t(2) * kBuf * sizeof(double);   // the callers' A and E fit in it too

struct Scratch {
    double2 cs[2][32];                    // (c, s) of a round's seats, by round parity
    double up[2][kGroups * SP], down[2][kGroups * SP];   // entries of E on their way to the next lower / higher seat group
    double lam[SP];                       // the diagonal, by index, when the sweeps are done
    double red[kWarps];
};

// sum over the worker threads' v (the rotation warp's is not counted); all threads call
__device__ __forceinline__ double block_sum(double v, double* red) {
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    const int warp = threadIdx.x >> 5;
    if ((threadIdx.x & 31) == 0 && warp < kWarps) red[warp] = v;
    __syncthreads();
    double r = red[0];
    for (int k = 1; k < kWarps; ++k) r += red[k];
    __syncthreads();
    return r;
}

// the index at a position in round 0 (and after every whole sweep)
__device__ __forceinline__ int index_at(int pos) {
    if (pos < 32) return pos == 0 ? SP - 1 : pos;
    return pos == 32 ? 0 : SP - 1 - (pos - 32);
}
// where the x / y of seat k goes after a round: row, and column
__device__ __forceinline__ int next_x(int k, int y_at) { return k == 0 ? 0 : (k == 1 ? y_at : k - 1); }
__device__ __forceinline__ int next_y(int k, int y_at) { return k == 31 ? 31 : y_at + k + 1; }
// seats k >= first_xp(r) have x < y, so x is their p; in the others y is
__device__ __forceinline__ int first_xp(int r) { return r <= 31 ? r + 1 : SP - 1 - r; }

// One pair of entries through a rotation, the p and the q result.  The roundings are spelled out: the
// rotation warp and the workers form the same entry independently, and the bits must agree.
__device__ __forceinline__ double rot_p(double2 r, double a, double b) { return fma(r.x, a, -__dmul_rn(r.y, b)); }
__device__ __forceinline__ double rot_q(double2 r, double a, double b) { return fma(r.y, a, __dmul_rn(r.x, b)); }

// rotation that annihilates a_pq: (c, s) and t = tan(theta)
__device__ __forceinline__ double2 rotation(double apq, double app, double aqq, double& t) {
    double c = 1.0, s = 0.0;
    t = 0.0;
    if (fabs(apq) >= 1e-300) {
        // t = tan(theta) of the smaller rotation, tau = (a_qq - a_pp) / (2 a_pq):
        // t = sign(tau) / (|tau| + sqrt(1 + tau^2)) = 2 a_pq sign(d) / (|d| + sqrt(d^2 + 4 a_pq^2)), d = a_qq - a_pp
        const double d = aqq - app;
        const double tt = 2.0 * apq / (fabs(d) + sqrt(fma(4.0 * apq, apq, __dmul_rn(d, d))));
        t = d >= 0.0 ? tt : -tt;
        c = rsqrt(fma(t, t, 1.0));
        s = t * c;
    }
    return make_double2(c, s);
}

// A worker's eight seats (kSeats) of one row of E through their rotations.  kRole: x is the p of 0 no seat, 1 every seat,
// 2 the seats k >= first.
template <int kRole>
__device__ __forceinline__ void rotate_seats(double (&ex)[kSeats], double (&ey)[kSeats], const double2* cs, int first) {
#pragma unroll
    for (int k = 0; k < kSeats; ++k) {
        const double2 q = cs[k];
        const double x = ex[k], y = ey[k];
        if (kRole == 1 || (kRole == 2 && k >= first)) {
            ex[k] = rot_p(q, x, y);
            ey[k] = rot_q(q, x, y);
        } else {
            ey[k] = rot_p(q, y, x);
            ex[k] = rot_q(q, y, x);
        }
    }
}

// What a worker keeps through all rounds: its part of E, and the offsets of its column and rows of A and of
// where they move to.
struct Worker {
    double ex[kSeats], ey[kSeats];
    int cx, cy, tx, ty;                                // column of x_J and y_J, J = lane, and where they go
    int rx[kBlocks], ry[kBlocks], sx[kBlocks], sy[kBlocks];   // rows of x_I and y_I of its blocks, and where they go
    int xe;                                            // its place in the entries of E passed on
};
// keep a value in its register: recomputing the offsets every round doubled the round's instructions
__device__ __forceinline__ void pin(int& x) { asm volatile("" : "+r"(x)); }

// Workers: apply round r to E (registers) and A (cur -> nxt).  `in` is the parity that the round's inputs have.
__device__ __forceinline__ void worker_round(Worker& w, const double* cur, double* nxt, Scratch& js, int in, int r, int wp, int lane,
                                             bool moved) {
    const double2* cs = js.cs[in];
    const int first = first_xp(r);
    {   // E first: the rotation warp's few loads then go ahead of the workers' many
        const int eh = wp >> 1;
        if (moved) {                                   // the entries that the last round passed on
            if (eh < kGroups - 1) w.ex[kSeats - 1] = js.up[in][w.xe];
            if (eh > 0) w.ey[0] = js.down[in][w.xe];
        }
        const int f = first - kSeats * eh;
        if (f >= kSeats) rotate_seats<0>(w.ex, w.ey, cs + kSeats * eh, f);
        else if (f <= 0) rotate_seats<1>(w.ex, w.ey, cs + kSeats * eh, f);
        else rotate_seats<2>(w.ex, w.ey, cs + kSeats * eh, f);
        if (eh > 0) js.up[in ^ 1][w.xe - SP] = w.ex[0];
        if (eh < kGroups - 1) js.down[in ^ 1][w.xe + SP] = w.ey[kSeats - 1];
        const double x0 = w.ex[0], x1 = w.ex[1], y_last = w.ey[kSeats - 1];
#pragma unroll
        for (int k = 0; k < kSeats - 1; ++k) w.ex[k] = w.ex[k + 1];
        if (eh == 0) w.ex[0] = x0;                     // 63 stays in seat 0
        w.ex[kSeats - 1] = y_last;                     // seat 31's x (the other groups' comes from above)
#pragma unroll
        for (int k = kSeats - 1; k > 0; --k) w.ey[k] = w.ey[k - 1];
        w.ey[0] = x1;                                  // seat 0's y (the other groups' comes from below)
    }
    const bool xc = lane >= first;
    const int pc = xc ? w.cx : w.cy, qc = xc ? w.cy : w.cx, pt = xc ? w.tx : w.ty, qt = xc ? w.ty : w.tx;
    const double2 rJ = cs[lane];
#pragma unroll
    for (int i = 0; i < kBlocks; ++i) {                // blocks (I, J) of A, J = lane
        const int I = wp + kWarps * i;
        const bool xr = I >= first;
        const int pr = xr ? w.rx[i] : w.ry[i], qr = xr ? w.ry[i] : w.rx[i];
        const double2 rI = cs[I];
        const double a = cur[pr + pc], b = cur[pr + qc], c = cur[qr + pc], d = cur[qr + qc];
        const double m0 = rot_p(rJ, a, b), m1 = rot_q(rJ, a, b);      // [a b; c d] R_J
        const double m2 = rot_p(rJ, c, d), m3 = rot_q(rJ, c, d);
        const int sp = xr ? w.sx[i] : w.sy[i], sq = xr ? w.sy[i] : w.sx[i];
        if (I != lane) {                                             // R_I^T (...); the rotation warp writes the diagonal blocks
            nxt[sp + pt] = rot_p(rI, m0, m2);
            nxt[sp + qt] = rot_p(rI, m1, m3);
            nxt[sq + pt] = rot_q(rI, m0, m2);
            nxt[sq + qt] = rot_q(rI, m1, m3);
        }
    }
}

// The rotation warp's round r, seat k = lane: the rotations of round r + 1.  dx, dy: the diagonal entries of the seat's
// occupants after round r, moved on here to round r + 1's occupants.
__device__ __forceinline__ void ahead_round(double& dx, double& dy, const double* cur, double* nxt, const double2* cs, double2* cs_next,
                                            int r, int k) {
    const int first = first_xp(r), next = first_xp(r + 1 < SP - 1 ? r + 1 : 0);
    // the next occupants' seats in this round, and whether they are its p: x comes from seat k + 1 (seat 31's is
    // its own y, seat 0's stays), y from seat k - 1 (seat 0's is seat 1's x)
    const int sx = k == 0 ? 0 : (k == 31 ? 31 : k + 1), sy = k == 0 ? 1 : k - 1;
    const bool x_is_p = (sx >= first) == (k != 31), y_is_p = (sy >= first) == (k == 0);
    const bool xp = k >= next;                         // the row of a_pq is the smaller index
    const int sr = xp ? sx : sy, sc = xp ? sy : sx;
    const bool rp = xp ? x_is_p : y_is_p, cp = xp ? y_is_p : x_is_p;
    const int pr = (sr >= first ? sr : 32 + sr) * kPitch, qr = (sr >= first ? 32 + sr : sr) * kPitch;
    const int pc = sc >= first ? sc : kYCol + sc, qc = sc >= first ? kYCol + sc : sc;
    const double2 rI = cs[sr], rJ = cs[sc];
    const double a = cur[pr + pc], b = cur[pr + qc], c = cur[qr + pc], d = cur[qr + qc];
    const double up = __shfl_down_sync(0xffffffffu, dx, 1), down = __shfl_up_sync(0xffffffffu, dy, 1);
    const double nx = k == 0 ? dx : (k == 31 ? dy : up), ny = k == 0 ? up : down;
    // rot_p or rot_q by choice of the coefficients
    const double c0 = cp ? rJ.x : rJ.y, c1 = cp ? -rJ.y : rJ.x, r0 = rp ? rI.x : rI.y, r1 = rp ? -rI.y : rI.x;
    const double u = fma(c0, a, __dmul_rn(c1, b)), v = fma(c0, c, __dmul_rn(c1, d));
    const double apq = fma(r0, u, __dmul_rn(r1, v));
    const double app = xp ? nx : ny, aqq = xp ? ny : nx;
    double t;
    cs_next[k] = rotation(apq, app, aqq, t);
    // this round's diagonal blocks
    nxt[next_x(k, 32) * kPitch + next_y(k, kYCol)] = 0.0;
    nxt[next_y(k, 32) * kPitch + next_x(k, kYCol)] = 0.0;
    nxt[k * (kPitch + 1)] = nx;
    nxt[(32 + k) * kPitch + kYCol + k] = ny;
    const double np = fma(-t, apq, app), nq = fma(t, apq, aqq);
    dx = xp ? np : nq;
    dy = xp ? nq : np;
}

// sm (kSmem bytes) holds A (symmetric, [64][LD]) and after it E ([64][LD]).  A is diagonalised, E multiplied by
// the rotations (start it at the identity, or at a warm-start basis with A already rotated into it).  On
// return js.lam holds the diagonal and E is where it was; A is lost.  All kThreads threads call.
__device__ __forceinline__ void sweeps(double* sm, Scratch& js, int max_sweeps) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int wp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const bool worker = wp < kWarps;
    // a warp holds one seat group of 32 rows of E, so which entry of a pair is its p is the same for all lanes
    const int eh = (wp >> 1) & (kGroups - 1), er = 32 * (wp & 1) + lane;
    double* E = sm + SP * LD + er * LD;
    Worker w;
#pragma unroll
    for (int k = 0; k < kSeats; ++k) {
        w.ex[k] = E[index_at(kSeats * eh + k)];
        w.ey[k] = E[index_at(32 + kSeats * eh + k)];
    }
    w.cx = lane; w.cy = kYCol + lane; w.tx = next_x(lane, kYCol); w.ty = next_y(lane, kYCol);
    w.xe = SP * eh + er;
    pin(w.cx); pin(w.cy); pin(w.tx); pin(w.ty); pin(w.xe);
#pragma unroll
    for (int i = 0; i < kBlocks; ++i) {
        const int I = (wp & (kWarps - 1)) + kWarps * i;
        w.rx[i] = I * kPitch; w.ry[i] = (32 + I) * kPitch; w.sx[i] = next_x(I, 32) * kPitch; w.sy[i] = next_y(I, 32) * kPitch;
        pin(w.rx[i]); pin(w.ry[i]); pin(w.sx[i]); pin(w.sy[i]);
    }
    // A by position, into the first buffer (it overlays the callers' A and E)
    double mine[SP2 / kWorkers];
    if (worker)
#pragma unroll
        for (int i = 0; i < SP2 / kWorkers; ++i) {
            const int e = tid + kWorkers * i;
            mine[i] = sm[index_at(e >> 6) * LD + index_at(e & 63)];
        }
    __syncthreads();
    if (worker)
#pragma unroll
        for (int i = 0; i < SP2 / kWorkers; ++i) {
            const int e = tid + kWorkers * i, j = e & 63;
            sm[(e >> 6) * kPitch + (j < 32 ? j : j - 32 + kYCol)] = mine[i];
        }
    int par = 0;                                       // parity of the round to apply: the buffer that holds A
    double dx = 0.0, dy = 0.0;                         // rotation warp: the seat's diagonal after that round
    bool moved = false;
    __syncthreads();
    for (int sweep = 0; sweep < max_sweeps; ++sweep) {
        const double* cur = sm + (par ? kBuf : 0);
        double off = 0.0, tot = 0.0;
        if (worker)
            for (int e = tid; e < SP2; e += kWorkers) {
                const int i = e >> 6, j = e & 63;
                const double v = cur[i * kPitch + (j < 32 ? j : j - 32 + kYCol)], x = v * v;
                tot += x;
                if (i != j) off += x;
            }
        off = block_sum(off, js.red);
        tot = block_sum(tot, js.red);
        if (off <= 1e-30 * tot || off == 0.0) break;
        if (!moved && !worker) {                       // round 0's rotations from A itself
            const bool xp = lane >= first_xp(0);
            const int pr = (xp ? lane : 32 + lane) * kPitch, qr = (xp ? 32 + lane : lane) * kPitch;
            const int pc = xp ? lane : kYCol + lane, qc = xp ? kYCol + lane : lane;
            const double apq = cur[pr + qc], app = cur[pr + pc], aqq = cur[qr + qc];
            double t;
            js.cs[par][lane] = rotation(apq, app, aqq, t);
            const double np = fma(-t, apq, app), nq = fma(t, apq, aqq);
            dx = xp ? np : nq;
            dy = xp ? nq : np;
        }
        for (int r = 0; r < SP - 1; ++r) {
            __syncthreads();                           // A of this round, its rotations and the other buffer are ready
            if (worker) {
                if (par == 0) worker_round(w, sm, sm + kBuf, js, 0, r, wp, lane, moved);
                else worker_round(w, sm + kBuf, sm, js, 1, r, wp, lane, moved);
            } else {
                if (par == 0) ahead_round(dx, dy, sm, sm + kBuf, js.cs[0], js.cs[1], r, lane);
                else ahead_round(dx, dy, sm + kBuf, sm, js.cs[1], js.cs[0], r, lane);
            }
            moved = true;
            par ^= 1;
        }
        __syncthreads();                               // the sweep's last round is complete
    }
    const double* cur = sm + (par ? kBuf : 0);
    if (tid < SP) js.lam[index_at(tid)] = cur[tid * kPitch + (tid < 32 ? tid : tid - 32 + kYCol)];
    if (worker && moved) {
        if (eh < kGroups - 1) w.ex[kSeats - 1] = js.up[par][w.xe];
        if (eh > 0) w.ey[0] = js.down[par][w.xe];
    }
    __syncthreads();                                   // A has been read: E's place is free
    if (worker)
#pragma unroll
        for (int k = 0; k < kSeats; ++k) {             // a whole number of sweeps: the seats of round 0 again
            E[index_at(kSeats * eh + k)] = w.ex[k];
            E[index_at(32 + kSeats * eh + k)] = w.ey[k];
        }
    __syncthreads();
}

// ------------------------------------------------------------------ symmetric form
// The same sweeps on half of A, for callers that do not need the bits of the form above: an entry between two
// occupants is kept once.  Entries are stored by the distance of their seats, S[kind][d][J] between seats I = J + d mod 32
// and J, d = 1 .. 16 (16: J < 16), kind = 2 (y at I) + (y at J), so a warp's loads are 32 consecutive entries; where an
// entry moves with its occupants is fixed, and looked up once.  The pivot of the next round, the entry of two
// occupants of one seat, goes to S[0][0][seat].  The x of a seat is always the p of its rotation.
// A round then moves about 600 wavefronts through shared memory instead of 1060, and the chain of the rotations bounds it:
// 1000 cycles instead of 1540.  61 states, 2 to 3 matrices: 398 -> 265 us (with rotation() 279; with the worker's loads
// all ahead of E 310, the rotation warp's wait behind them).  Codon generators, 400 drawn: departure from orthogonality
// 3.3e-15 on average (worst 5.5e-15), residual 2.5e-15 (5.6e-15) of the largest entry; with sweeps() 4.0e-15 (6.2e-15)
// and 2.8e-15 (6.1e-15).
constexpr int kSymKind = 17 * 32;                      // entries of one kind
constexpr int kSymBuf = 4 * kSymKind;
constexpr size_t kSymSmem = (size_t(2) * SP * LD + 2 * kSymBuf) * sizeof(double);     // the callers' A and E, two buffers of S
constexpr int kSymBlocks = 16 / kWarps;                // distances a worker warp updates

// an occupant's place: 2 seat + (is y); where it goes after a round
__device__ __forceinline__ int sym_next(int at) {
    const int k = at >> 1;
    if (at & 1) return k == 31 ? 2 * 31 : at + 2;
    return k == 0 ? 0 : (k == 1 ? 1 : at - 2);
}
// where the entry between two places is kept
__device__ __forceinline__ int sym_slot(int a, int b) {
    int I = a >> 1, J = b >> 1, d = (I - J) & 31;
    if (d == 0) return I;
    if (d > 16 || (d == 16 && J >= 16)) {
        const int x = a; a = b; b = x;
        J = I;
        d = 32 - d;
    }
    return (2 * (a & 1) + (b & 1)) * kSymKind + 32 * d + J;
}

// The rotation that annihilates a_pq, by the double angle: with h = d^2 + 4 a_pq^2, d = a_qq - a_pp, cos 2theta = |d| / sqrt(h),
// c^2 = (1 + cos 2theta) / 2 and s = a_pq sign(d) / (c sqrt(h)); two reciprocal square roots in a row where
// rotation() has a square root, a divide and a reciprocal square root.  One Newton step makes c^2 + s^2 = 1 to the
// last bits.  Entries below 1e-150 (squares that the sweeps' test cannot see) count as zero.
__device__ __forceinline__ double2 rotation_sym(double apq, double app, double aqq, double& t) {
    const double d = aqq - app, h = fma(4.0 * apq, apq, d * d);
    double c = 1.0, s = 0.0;
    t = 0.0;
    if (fabs(apq) >= 1e-150 && h <= 1e300) {
        const double r = rsqrt(h), c2 = fma(0.5 * fabs(d), r, 0.5), rc = rsqrt(c2);
        const double sa = (d >= 0.0 ? apq : -apq) * r;
        c = c2 * rc;
        s = sa * rc;
        t = s * rc;
        const double n = 0.5 * fma(s, s, fma(c, c, -1.0));
        c = fma(-n, c, c);
        s = fma(-n, s, s);
    }
    return make_double2(c, s);
}

// sm (kSymSmem bytes) holds A and E as for sweeps(), the results are the same: js.lam and E in place.
__device__ __forceinline__ void sweeps_sym(double* sm, Scratch& js, int max_sweeps) {
    const int tid = threadIdx.x, lane = tid & 31;
    const int wp = __shfl_sync(0xffffffffu, tid >> 5, 0);
    const bool worker = wp < kWarps;
    double* S = sm + 2 * SP * LD;
    const int eh = (wp >> 1) & (kGroups - 1), er = 32 * (wp & 1) + lane, xe = SP * eh + er;
    double* E = sm + SP * LD + er * LD;
    double ex[kSeats], ey[kSeats];
#pragma unroll
    for (int k = 0; k < kSeats; ++k) {
        ex[k] = E[index_at(kSeats * eh + k)];
        ey[k] = E[index_at(32 + kSeats * eh + k)];
    }
    // a place's index in round 0
    auto index_of = [](int at) { return index_at((at & 1) * 32 + (at >> 1)); };
    for (int e = tid; e < 2 * kSymBuf; e += kThreads) S[e] = 0.0;
    __syncthreads();
    double tot = 0.0;
    for (int e = tid; e < SP * SP; e += kThreads) {
        const int a = e >> 6, b = e & 63;
        if (a >= b) continue;
        const double v = sm[index_of(a) * LD + index_of(b)];
        S[sym_slot(a, b)] = v;
        tot += 2.0 * v * v;
    }
    if (tid < SP) { const double v = sm[tid * LD + tid]; tot = fma(v, v, tot); }
    // workers: the slots that their blocks' entries move to; the rotation warp: its next pivot's block and where a zero goes
    int to[kSymBlocks][4], from[kSymBlocks], zero = 0, ahead[4];
    double gx = 0.0, gy = 0.0, dx = 0.0, dy = 0.0;     // rotation warp: the seat's diagonal before and after the round to come
    bool xa = true, xb = false;                        // the next pivot is between an x and a y
#pragma unroll
    for (int i = 0; i < kSymBlocks; ++i) {
        const int d = 1 + (wp & (kWarps - 1)) + kWarps * i, I = (lane + d) & 31;
        from[i] = 32 * d + lane;
#pragma unroll
        for (int e = 0; e < 4; ++e)                    // (distance 16, J >= 16: zeros, kept where they are)
            to[i][e] = d == 16 && lane >= 16 ? e * kSymKind + from[i] : sym_slot(sym_next(2 * I + (e >> 1)), sym_next(2 * lane + (e & 1)));
#pragma unroll
        for (int e = 0; e < 4; ++e) pin(to[i][e]);
    }
    {
        const int k = lane, sa = k == 0 ? 0 : (k == 31 ? 31 : k + 1), sb = k == 0 ? 1 : k - 1;
        xa = k != 31;
        xb = k == 0;
        for (int e = 0; e < 4; ++e) ahead[e] = sym_slot(2 * sa + (e >> 1), 2 * sb + (e & 1));
        zero = sym_slot(sym_next(2 * k), sym_next(2 * k + 1));
        if (!worker) {
            gx = sm[index_at(k) * (LD + 1)];
            gy = sm[index_at(32 + k) * (LD + 1)];
        }
    }
    double part = worker ? tot : 0.0, rest = worker ? 0.0 : tot;
    for (int o = 16; o > 0; o >>= 1) rest += __shfl_xor_sync(0xffffffffu, rest, o);
    if (!worker && lane == 0) js.up[0][0] = rest;      // the rotation warp's share of the total
    tot = block_sum(part, js.red);
    tot += js.up[0][0];
    __syncthreads();
    int par = 0;                                       // parity of the round to apply: the buffer that holds it
    bool moved = false;
    for (int sweep = 0; sweep < max_sweeps; ++sweep) {
        const double* cur = S + (par ? kSymBuf : 0);
        double off = 0.0;
        if (worker)
            for (int e = tid; e < kSymBuf; e += kWorkers) off = fma(cur[e], cur[e], off);
        off = 2.0 * block_sum(off, js.red);
        if (off <= 1e-30 * tot || off == 0.0) break;
        if (!moved && !worker) {
            double t;
            const double a = cur[lane];
            js.cs[par][lane] = rotation_sym(a, gx, gy, t);
            dx = fma(-t, a, gx);
            dy = fma(t, a, gy);
        }
        for (int r = 0; r < SP - 1; ++r) {
            __syncthreads();                           // this round's entries and rotations, and the other buffer, are ready
            const double* A = S + (par ? kSymBuf : 0);
            double* B = S + (par ? 0 : kSymBuf);
            const double2* cs = js.cs[par];
            if (worker) {
                {   // E first: the rotation warp's few loads then go ahead of the workers' many
                    const double2* ce = cs + kSeats * eh;
                    if (moved) {                       // the entries of E that the last round passed on
                        if (eh < kGroups - 1) ex[kSeats - 1] = js.up[par][xe];
                        if (eh > 0) ey[0] = js.down[par][xe];
                    }
#pragma unroll
                    for (int k = 0; k < kSeats; ++k) {
                        const double2 q = ce[k];
                        const double x = ex[k], y = ey[k];
                        ex[k] = rot_p(q, x, y);
                        ey[k] = rot_q(q, x, y);
                    }
                    if (eh > 0) js.up[par ^ 1][xe - SP] = ex[0];
                    if (eh < kGroups - 1) js.down[par ^ 1][xe + SP] = ey[kSeats - 1];
                    const double x0 = ex[0], x1 = ex[1], y_last = ey[kSeats - 1];
#pragma unroll
                    for (int k = 0; k < kSeats - 1; ++k) ex[k] = ex[k + 1];
                    if (eh == 0) ex[0] = x0;
                    ex[kSeats - 1] = y_last;
#pragma unroll
                    for (int k = kSeats - 1; k > 0; --k) ey[k] = ey[k - 1];
                    ey[0] = x1;
                }
                const double2 rJ = cs[lane];
#pragma unroll
                for (int i = 0; i < kSymBlocks; ++i) {
                    const double2 rI = cs[(lane + 1 + wp + kWarps * i) & 31];
                    const double a = A[from[i]], b = A[from[i] + kSymKind], c = A[from[i] + 2 * kSymKind], d = A[from[i] + 3 * kSymKind];
                    const double m0 = rot_p(rJ, a, b), m1 = rot_q(rJ, a, b);
                    const double m2 = rot_p(rJ, c, d), m3 = rot_q(rJ, c, d);
                    B[to[i][0]] = rot_p(rI, m0, m2);
                    B[to[i][1]] = rot_p(rI, m1, m3);
                    B[to[i][2]] = rot_q(rI, m0, m2);
                    B[to[i][3]] = rot_q(rI, m1, m3);
                }
            } else {
                const int k = lane;
                const double2 ra = cs[k == 0 ? 0 : (k == 31 ? 31 : k + 1)], rb = cs[k == 0 ? 1 : k - 1];
                const double v0 = A[ahead[0]], v1 = A[ahead[1]], v2 = A[ahead[2]], v3 = A[ahead[3]];
                const double up = __shfl_down_sync(0xffffffffu, dx, 1), down = __shfl_up_sync(0xffffffffu, dy, 1);
                gx = k == 0 ? dx : (k == 31 ? dy : up);
                gy = k == 0 ? up : down;
                const double a0 = xa ? ra.x : ra.y, a1 = xa ? -ra.y : ra.x, b0 = xb ? rb.x : rb.y, b1 = xb ? -rb.y : rb.x;
                const double apq = fma(a0, fma(b0, v0, __dmul_rn(b1, v1)), __dmul_rn(a1, fma(b0, v2, __dmul_rn(b1, v3))));
                double t;
                js.cs[par ^ 1][k] = rotation_sym(apq, gx, gy, t);
                B[zero] = 0.0;
                dx = fma(-t, apq, gx);
                dy = fma(t, apq, gy);
            }
            moved = true;
            par ^= 1;
        }
        __syncthreads();                               // the sweep's last round is complete
    }
    if (!worker) {
        js.lam[index_at(lane)] = gx;
        js.lam[index_at(32 + lane)] = gy;
    } else {
        if (moved) {
            if (eh < kGroups - 1) ex[kSeats - 1] = js.up[par][xe];
            if (eh > 0) ey[0] = js.down[par][xe];
        }
#pragma unroll
        for (int k = 0; k < kSeats; ++k) {             // a whole number of sweeps: the seats of round 0 again
            E[index_at(kSeats * eh + k)] = ex[k];
            E[index_at(32 + kSeats * eh + k)] = ey[k];
        }
    }
    __syncthreads();
}

}  // namespace jac
}  // namespace h3g
