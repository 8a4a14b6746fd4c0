// kofm_sstep.cuh - the k-omega solve in two sweeps over the matrix per
// restart cycle (sm_100a).
//
// Algorithm: the reference's restarted "simpler GMRES" (GMRESSolver::solve,
// GMRESSolver.cpp:227-355; Walker & Zhou 1994) on the correction system
// A d = b' with the same restart loop, convergence test, truncation tests
// (diag(R) against relTol R(0,0), then |xi_k| >= rho), residual estimator
// and x = x0 + d.  What changes is how a cycle is computed.
//
// The rows are normalised by their diagonal, so A = I + N with N the four
// off-diagonals.  The Krylov space of A on r equals that of N, spanned by the
// powers p_0 = r, p_{j+1} = N p_j.  A cycle is
//   * one sweep that marches p_1 .. p_L through registers and sums the Gram
//     matrix G = P^T P of [p_0 .. p_L] on the way (ss_march<L, true>);
//   * the simpler GMRES in the (L+1)-dimensional coefficient space (one warp
//     per system): with A p_j = p_j + p_{j+1} every inner product of the
//     method is a combination of G's entries;
//   * one sweep that marches the powers again and adds d = sum c_j p_j to the
//     field (ss_march<M, false>).
// No power is ever written to memory: each sweep streams the four
// coefficients and p_0 (40 bytes a node), the second also the field.  The
// residual of the cycle's end, r - A d = sum e_j p_j, has the norm e^T G e, so
// the next restart's convergence test needs no sweep either: where it passes
// by more than the rounding of that sum, the second sweep adds d to the field
// at once.  Where it does not (tight tolerances, or a further restart), the
// second sweep keeps d, and a residual sweep forms b' - A d and its norm.
//
// L follows the cycle lengths seen so far (two more powers than the last such
// cycle used, kept per system across solves, for a solve's first cycle and for
// its later ones, which are shorter); a cycle whose tests have not fired by then
// is run again with the powers up to the Krylov dimension.
// In FP64 the truncation tests see rounding of the size the reference's own
// classical Gram-Schmidt has (both lose orthogonality like eps cond^2), so the
// cut of a converged cycle moves by a vector or two with the order of a sum, and
// with it the end residual, between about 1e-6 and 1e-9 ||b'|| (the tolerance is
// 1e-4).  In a running channel that is far below the fields' rounding; in the
// first solve of a loaded state it need not be, so that one takes its sums in a
// fixed order (sp_first_gram_kernel).
#pragma once
#include "kofm_gmres.cuh"

namespace kofm {

constexpr int SS_THREADS = 256;
constexpr int SS_WARPS = SS_THREADS / 32;
constexpr int SS_MAXL = KOFM_MAX_KRYLOV;                  // levels of one sweep
constexpr int SS_NG = (SS_MAXL + 1) * (SS_MAXL + 2) / 2;  // Gram entries per system
constexpr int SS_MINL = 4;                                // fewest powers of a first round

// What the second sweep does for a system (GmresSys::bmode).
enum SsApply : int {
    SS_B_NONE = 0,
    SS_B_FINAL,   // field += d (the solve has ended)
    SS_B_UPDATE,  // x = x + d (a residual sweep follows)
    SS_B_WRITE,   // field += x if a cycle was run, pointwise (the solve ended at a convergence test)
};

struct SsQueue {
    unsigned int count;  // blocks that have finished the sweep
    unsigned int pad;
};

struct SsArgs {
    KoSystem sys[2];
    void* field[2];           // omega, k (updated in place at the end): FP32, or FP64 when f64
    int f64;
    const int16_t* ntype;
    GmresControl* ctl;
    double* part;             // partial sums [2][maxu][SS_NG] (a unit's sums side by side)
    int maxu;
    GridBarrier* bar;
    SsQueue* queue;
    int* lhint;               // powers of a cycle's first sweep, kept across solves (0: K): [2] of a solve's
                              // first cycle, [2] of zeros for a loaded state's first solve, [2] of later cycles
    int nx, ny, P;
    long long D;
    int K;                    // Krylov dimension
    int max_restarts;
    double rel_tol, abs_tol;
    long long spin_limit;
    int launches;             // of an update
    // row ranges a strip is split into, by both systems' level counts + 1 (0: a
    // system with nothing to do): the Gram sweep and the update sweep
    short gram_rows[SS_MAXL + 2][SS_MAXL + 2];
    short upd_rows[SS_MAXL + 2][SS_MAXL + 2];
};

// Gram entry (i, j), i <= j, of one system: slot j (j + 1) / 2 + i.
__host__ __device__ constexpr int ss_gslot(int i, int j) { return j * (j + 1) / 2 + i; }

__host__ __device__ __forceinline__ int ss_hint_levels(int l, int K) {
    if (l <= 0 || l > K) l = K;
    return l < SS_MINL ? (K < SS_MINL ? K : SS_MINL) : l;
}

// ---- coefficient-space simpler GMRES (serial step) -------------------------------
// Scratch of one system's serial step.
struct SsCycleSmem {
    double G[(SS_MAXL + 1) * (SS_MAXL + 1)];
    double R[SS_MAXL * SS_MAXL];  // R(j, k) at j + k K
    double xi[SS_MAXL], rho[SS_MAXL + 1];  // rho[k]: the estimator before vector k
    int cap;  // vectors the cycle may build (numerical rank of the power basis)
};

// Smallest pivot of the unit-diagonal Gram Cholesky accepted for a level.
constexpr double SS_PIVOT_MIN = 1.0e-9;
// Rounding of the predicted residual's square, relative to the sum of the
// magnitudes of its terms (the Gram entries' own sums over the nodes).
constexpr double SS_PRED_EPS = 1.0e-13;

// Sum over each half of a warp: every lane of the half gets it, the same to the
// last bit (an addition that is not fused with the product a caller passes, or
// two lanes would round it differently and could take different branches).
__device__ __forceinline__ double ss_sum16(double x) {
#pragma unroll
    for (int off = 8; off > 0; off >>= 1) x = __dadd_rn(x, __shfl_xor_sync(0xffffffffu, x, off));
    return x;
}

// Numerical rank of the power basis p_0 .. p_L, one warp: Cholesky of the Gram
// scaled to a unit diagonal, whose j-th pivot is sin^2 of the angle between
// p_j and span(p_0 .. p_{j-1}).  Levels from the first pivot below SS_PIVOT_MIN
// on carry too few correct digits for the coefficient-space orthogonalisation
// (the monomial basis turns towards the dominant eigenvector as the operator's
// convective part grows).  Lane i holds row i.
__device__ __forceinline__ void ss_rank(SsCycleSmem& cs, int n) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    double sc = 0.0;
    if (lane < n) {
        const double gii = cs.G[lane * n + lane];
        sc = gii > 0.0 ? rsqrt(gii) : 0.0;
    }
    double row[SS_MAXL + 1];
#pragma unroll
    for (int k = 0; k <= SS_MAXL; ++k) {
        const double sk = __shfl_sync(FULL, sc, k);
        row[k] = lane < n && k < n ? cs.G[lane * n + k] * (sc * sk) : 0.0;
    }
    int rank = n;
#pragma unroll
    for (int j = 0; j <= SS_MAXL; ++j) {
        if (j >= n) break;
        const double p = __shfl_sync(FULL, row[j], j);
        if (!(p > SS_PIVOT_MIN)) { rank = j; break; }
        const double l = row[j] * rsqrt(p);
#pragma unroll
        for (int k = j + 1; k <= SS_MAXL; ++k) row[k] -= l * __shfl_sync(FULL, l, k);
    }
    if (lane == 0) cs.cap = rank - 1 < 1 ? 1 : rank - 1;  // vector k uses levels up to k + 1
}

// The cycle's vectors in coefficient space, one warp: lane i holds coefficient
// i (on p_i) of every vector and row i of G.  With A p_j = p_j + p_{j+1}, w = A
// z is a shift, the inner products of classical Gram-Schmidt are w^T G v_j
// with the unmodified w (the reference's order, so that the truncation tests
// meet rounding of the reference's kind), and v_k = w / ||w||.  Stops at the
// first vector that the reference's tests refuse (GMRESSolver.cpp:300-330):
// diag(R) below rel_tol R(0, 0), or |xi_k| >= rho.  Latency-bound: a chain of a
// shift, one product with G, two sums over the lanes and a square root per
// vector.  The warp's halves do the same work, so that every lane holds what
// the tests read.
// ORDERED: with the estimator, the quotients and the order of the sums as the
// reference's formulas have them (GMRESSolver.cpp:300-330), for sums whose
// rounding decides the result (sp_first_gram_kernel); in every solve that would
// be 3 us of a step's 57 at 256x64.
struct SsCycle {
    double V[SS_MAXL];  // this lane's coefficient of v_0 .. v_{built-1}
    int built;          // vectors built
    int cut;            // 0: none (all L vectors passed), 1: diag(R), 2: xi, 3: all K built
};
template <bool ORDERED>
__device__ __forceinline__ void ss_cycle(SsCycle& c, SsCycleSmem& cs, int L, int K, double rel_tol, double rinv) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 15;
    const int n = L + 1;
    double g[SS_MAXL + 1], GV[SS_MAXL];
#pragma unroll
    for (int j = 0; j <= SS_MAXL; ++j) g[j] = lane < n && j < n ? cs.G[lane * n + j] : 0.0;
    double rho = 1.0, r00 = 0.0;
    c.built = 0;
    c.cut = 0;
#pragma unroll
    for (int k = 0; k < SS_MAXL; ++k) {
        if (k >= L || k >= K || c.cut) break;
        // w = A z, z = r / rho0 = rinv p_0 (k = 0) or v_{k-1}
        const double z = k == 0 ? (lane == 0 ? rinv : 0.0) : c.V[k > 0 ? k - 1 : 0];
        const double zm = __shfl_up_sync(FULL, z, 1, 16);
        double w = lane < n ? (lane == 0 ? z : z + zm) : 0.0;
        double a0 = 0.0, a1 = 0.0;
#pragma unroll
        for (int j = 0; j <= SS_MAXL; ++j) {
            const double wj = __shfl_sync(FULL, w, j);
            if (!ORDERED && (j & 1)) a1 += g[j] * wj;
            else if (!ORDERED || j < n) a0 += g[j] * wj;
        }
        double Gw = a0 + a1;
        double h[SS_MAXL];
#pragma unroll
        for (int j = 0; j < k; ++j) h[j] = ss_sum16(w * GV[j]);
#pragma unroll
        for (int j = 0; j < k; ++j) {
            w -= h[j] * c.V[j];
            Gw -= h[j] * GV[j];
        }
        const double nk2 = ss_sum16(w * Gw);
        double inv, nk;  // a vanishing direction cuts (diag test)
        if (ORDERED) {
            nk = nk2 > 0.0 ? sqrt(nk2) : 0.0;
            inv = nk > 0.0 ? 1.0 / nk : 0.0;
        } else {
            inv = nk2 > 0.0 ? rsqrt(nk2) : 0.0;
            nk = nk2 > 0.0 ? nk2 * inv : 0.0;
        }
        c.V[k] = w * inv;
        GV[k] = Gw * inv;
        const double xi = rinv * __shfl_sync(FULL, GV[k], 0, 16);  // <r / rho0, v_k>
        if (k == 0) r00 = nk;
        if (lane == 0) {
#pragma unroll
            for (int j = 0; j < k; ++j) cs.R[j + k * K] = h[j];
            cs.R[k + k * K] = nk;
            cs.xi[k] = xi;
            cs.rho[k] = rho;
        }
        c.built = k + 1;
        const double x = fabs(xi);
        if (nk < rel_tol * r00) c.cut = 1;
        else if (x >= rho) c.cut = 2;
        else {
            rho = ORDERED ? rho * sin(acos(xi / rho)) : sqrt((rho - x) * (rho + x));
            if (k == K - 1) c.cut = 3;
        }
    }
    if (lane == 0) cs.rho[c.built] = rho;
    __syncwarp();
}

// Start of a system's serial step after a Gram sweep of L levels, every second
// warp: t holds G(i, j) of p_0 .. p_L (slots ss_gslot).  Restart 0's first
// sweep also takes the restart-0 convergence test from G(0, 0) = ||b'||^2
// (GMRESSolver::solve's checkConvergence).
__device__ __forceinline__ void ss_gram_begin(const SsArgs& a, GmresSys& S, const double* t, int L, SsCycleSmem& cs) {
    const int lane = threadIdx.x & 31, part = threadIdx.x >> 6;
    const int n = L + 1;
    for (int e = lane + 32 * part; e < n * n; e += 16 * SS_WARPS) {
        const int i = e / n, j = e - i * n;
        cs.G[e] = t[i <= j ? ss_gslot(i, j) : ss_gslot(j, i)];
    }
    // (a cut by diag(R) indexes R with another stride and meets entries that no
    // vector writes: they are 0, as in the reference)
    for (int e = lane + 32 * part; e < a.K * a.K; e += 16 * SS_WARPS) cs.R[e] = 0.0;
    if (part == 0 && lane == 0) {
        const double rho0 = sqrt(t[0]);
        S.powers += L;
        if (S.restarts == 0) {
            S.norm_rhs = rho0;
            S.rho0 = rho0;
            S.restarts = 1;
            const double resid = rho0 / rho0;
            if (isnan(resid) || S.inject) { S.nan = 1; S.active = 0; }
            else if (resid <= a.rel_tol || rho0 <= a.abs_tol) { S.conv = 1; S.active = 0; }
            else S.cycles += 1;
        }
        if (!S.active) {
            S.lto = 0;
            S.bmode = SS_B_WRITE;
        } else {
            S.rho0 = rho0;
            S.rinv = 1.0 / rho0;
        }
    }
}

// End of the serial step: the cut, the update coefficients on p_0 .. p_L into
// S.h, and what the update sweep does with them.  A cycle whose tests have
// not fired asks for all powers (ext).
__device__ __forceinline__ void ss_gram_end(const SsArgs& a, GmresSys& S, int s, int L, SsCycleSmem& cs, SsCycle& c) {
    const unsigned FULL = 0xffffffffu;
    const int lane = threadIdx.x & 31;
    const int n = L + 1, K = a.K;
    // the powers past level cap are numerically dependent on the earlier ones:
    // the cycle ends with the vectors built (back-substitution as for a xi
    // cut), and the next restart goes on from its residual
    int kk, full = K;
    if (c.built > cs.cap || (!c.cut && c.built == cs.cap && cs.cap < L && cs.cap < K)) {
        c.built = kk = cs.cap;
        c.cut = 4;
    } else {
        kk = c.cut == 3 ? K : c.built - 1;
        if (c.cut == 1) full = kk;
    }
    if (!c.cut) {
        if (lane == 0) {
            S.ext = 1;  // the cycle again with all powers
            S.lto = K;
        }
        __syncwarp();
        return;
    }
    // back-substitution with R indexed by stride `full` (GMRESSolver.cpp:330-343);
    // coefficient 0 is applied even when the cycle is cut at k = 0, as the
    // reference's update does (its xi(0) then unscaled)
    double y = lane < c.built ? cs.xi[lane] : 0.0;
    double cc = kk == 0 && lane == 0 ? y : 0.0;
    const double inv = lane < kk ? 1.0 / cs.R[lane + lane * full] : 0.0;
    for (int j = kk - 1; j >= 0; --j) {
        const double x = __shfl_sync(FULL, y * inv, j);
        if (lane == j) cc = x * S.rho0;
        else if (lane < j) y -= cs.R[lane + j * full] * x;
    }
    double cp = __shfl_sync(FULL, cc, 0) * (lane == 0 ? S.rinv : 0.0);
#pragma unroll
    for (int j = 1; j < SS_MAXL; ++j) {
        const double x = __shfl_sync(FULL, cc, j);
        if (j < kk) cp += x * c.V[j - 1];
    }
    // the cycle's end: r - A d = sum e_j p_j, e_j = delta_j0 - c_j - c_{j-1}
    const double cm = __shfl_up_sync(FULL, cp, 1);
    const double e = lane < n ? (lane == 0 ? 1.0 - cp : -(cp + cm)) : 0.0;
    double g = 0.0, ga = 0.0;
#pragma unroll
    for (int j = 0; j <= SS_MAXL; ++j) {
        const double ej = __shfl_sync(FULL, e, j);
        if (j < n && lane < n) {
            const double x = cs.G[lane * n + j] * ej;
            g += x;
            ga += fabs(x);
        }
    }
    const double rr = ss_sum16(e * g), mag = ss_sum16(fabs(e) * ga);
    if (lane < SS_MAXL) S.h[lane] = lane < n ? cp : 0.0;
    if (lane == 0) {
        S.kk = kk;
        // xi tests taken: those of a xi cut include the vector refused
        S.iters += c.cut == 1 ? kk : c.built;
        S.update_terms += kk;
        S.rho = cs.rho[c.cut == 1 || c.cut == 2 ? c.built - 1 : c.built];
        S.prev_err = fabs(S.rho * S.rho0 / S.norm_rhs);
        S.done = 1;
        S.lev = L;
        S.ext = 0;
        S.lto = 0;
        S.vecs += c.built;
        S.vec_index_sum += c.built * (c.built - 1) / 2;
        int nl = c.built + 2;
        nl = nl > K ? K : nl;
        __stcg(a.lhint + s + (S.rst ? 4 : 0), nl);
        if (!S.rst) S.lnext = nl;
        // the next restart's test (GMRESSolver.cpp:248-256), where it is certain
        const int next = S.rst + 1;
        const double thr = fmax(a.rel_tol * S.norm_rhs, a.abs_tol);
        if (next >= a.max_restarts) {
            S.active = 0;  // iteration cap: the loop ends without a test
            S.bmode = SS_B_FINAL;
        } else if (sqrt(rr + SS_PRED_EPS * mag) <= thr * (1.0 - 1.0e-9)) {
            S.restarts += 1;
            S.rho0 = sqrt(fmax(rr, 0.0));
            S.conv = 1;
            S.active = 0;
            S.bmode = SS_B_FINAL;
        } else {
            S.bmode = SS_B_UPDATE;
        }
        // the update sweep: p_0, the coefficients where powers are needed, the
        // correction in after the first cycle; the field in and out with the
        // flags, or the correction out
        S.abytes += 8.0 + (kk > 1 ? 32.0 : 0.0) + (S.rst > 0 ? 8.0 : 0.0);
        S.abytes += S.bmode == SS_B_FINAL ? (a.f64 ? 18.0 : 10.0) : 8.0;
    }
    __syncwarp();
}

// One system's serial step after the residual sweep: rr = ||b' - A d||^2, the
// residual of the next restart (GMRESSolver.cpp:248-256).
__device__ __forceinline__ void ss_resid_step(const SsArgs& a, GmresSys& S, int s, double rr) {
    S.abytes += 56.0;  // the correction, four coefficients and b' in, r out, per node
    S.rho0 = sqrt(rr);
    S.restarts += 1;
    const double resid = S.rho0 / S.norm_rhs;
    if (isnan(resid)) { S.nan = 1; S.active = 0; }
    else if (resid <= a.rel_tol || S.rho0 <= a.abs_tol) { S.conv = 1; S.active = 0; }
    else S.cycles += 1;
    S.rst += 1;
    S.ready = 0;
    S.lto = S.active ? ss_hint_levels(__ldcg(a.lhint + 4 + s), a.K) : 0;
    if (!S.active) S.bmode = SS_B_WRITE;
}

// (the words in flight and their arrival are separate, so that other loads can
// be issued between)
struct SsSysWord {
    static constexpr int NW = (int)(sizeof(GmresSys) / 8);
    unsigned long long w;
    __device__ __forceinline__ void load(const GmresControl* ctl, int s) {
        static_assert(NW <= SS_THREADS && sizeof(GmresSys) % 8 == 0, "one word a thread");
        if ((int)threadIdx.x < NW) w = __ldcg(reinterpret_cast<const unsigned long long*>(&ctl->sys[s]) + threadIdx.x);
    }
    __device__ __forceinline__ void put(GmresSys& dst) const {
        if ((int)threadIdx.x < NW) reinterpret_cast<unsigned long long*>(&dst)[threadIdx.x] = w;
    }
};
__device__ __forceinline__ void sp_sys_load(const GmresControl* ctl, int s, GmresSys& dst) {
    constexpr int NW = (int)(sizeof(GmresSys) / 8);
    const unsigned long long* src = reinterpret_cast<const unsigned long long*>(&ctl->sys[s]);
    unsigned long long* d = reinterpret_cast<unsigned long long*>(&dst);
    for (int i = threadIdx.x; i < NW; i += blockDim.x) d[i] = __ldcg(src + i);
}

__device__ __forceinline__ void sp_sys_store(GmresControl* ctl, int s, const GmresSys& src) {
    constexpr int NW = (int)(sizeof(GmresSys) / 8);
    const unsigned long long* sp = reinterpret_cast<const unsigned long long*>(&src);
    unsigned long long* d = reinterpret_cast<unsigned long long*>(&ctl->sys[s]);
    for (int i = threadIdx.x; i < NW; i += blockDim.x) __stcg(d + i, sp[i]);
}

// ---- the sweeps -----------------------------------------------------------------
// A unit is one system's rows [ya, yb) of a strip of SS_THREADS columns, the
// outer L on each side halo.  Thread t holds column x0 - L + t (periodic);
// level j is valid on threads j .. SS_THREADS - 1 - j.  Step i takes p_0 and the
// coefficients at row tau = ya - L + i and computes level j at row tau - j
// from level j-1 at rows tau-j-1, tau-j (and its x neighbours, which the step
// before left in shared memory) and tau-j+1: a skewed wavefront, so that a row
// is read once for all levels.
//
// What bounds it: a step's latency.  40 bytes a node are read, which HBM would
// deliver in about 430 cycles a step of 256 columns; the FP64 pipe needs about
// 16 L cycles for the powers and 2 (L+1)(L+2) for the Gram sums; but 8 warps of
// up to 240 registers leave two warps to a scheduler, and a step is a chain
// (neighbours from shared memory, L dependent FMAs, the row back to shared
// memory, one barrier) that they only partly fill.  So everything is kept off
// that chain: a producer warp of its own fetches the rows ahead by bulk copies
// into a shared-memory ring (issued by one of the marching warps they held it,
// and through the barrier the block, for 350 to 500 cycles a step; as 8-byte
// cp.async by every thread they ran out of L1 beside this much shared memory),
// two levels' neighbours come by one 16-byte load, and what needs no other
// warp (the Gram sums of a complete row, the next row's inputs) follows the
// barrier.  The producer's warpgroup hands its registers to the marching ones
// (setmaxnreg: 128 x 24 + 256 x 240 = 384 x 168).
//
// The step loop is unrolled so that all register windows are circular buffers
// with compile-time slots: level j's row y stays in registers until the Gram
// sums of row y are formed (L - j steps later); the compiler keeps each value
// exactly that long.  From 7 levels on, the registers keep three rows and the
// older values wait in shared memory (the far history).

// Dynamic shared memory of a march: the ring, the rows that the threads'
// x neighbours read (the newest values of two levels side by side, per step
// parity, one column more on each side), and the far history of a Gram sweep
// of 7 and more levels (one column per thread).
__host__ __device__ constexpr int ss_row_bytes() { return (SS_THREADS + 2) * 16; }
__host__ __device__ constexpr int ss_nb_bytes(int L) { return 2 * ((L + 1) / 2) * ss_row_bytes(); }
constexpr int SS_FAR = 7;  // levels from which a Gram sweep keeps a far history
// Shared-memory rings of the far history: a ring has one slot a step of the
// unrolled loop (U), a level k occupies L - k of them behind its write
// position, and levels whose spans fit side by side share a ring.
struct SsFar {
    int ring[SS_MAXL + 1], shift[SS_MAXL + 1], rings;
    __host__ __device__ constexpr SsFar(int L) : ring{}, shift{}, rings(0) {
        const int U = (L + 3) / 3 * 3;
        int used[SS_MAXL + 1] = {};
        for (int k = 0; k + 3 <= L; ++k) {
            const int need = L - k;  // read before the slot is written again
            int r = 0;
            while (r < rings && used[r] + need > U) ++r;
            if (r == rings) ++rings;
            ring[k] = r;
            // spans run backwards from the write position: [pos - need + 1, pos]
            shift[k] = used[r] + need;
            used[r] += need;
        }
    }
};
__host__ __device__ constexpr int ss_far_bytes(int L) {
    return L < SS_FAR ? 0 : SsFar(L).rings * ((L + 3) / 3 * 3) * 8 * SS_THREADS;
}
// rows of the ring (the copies run one row less ahead): 12, or what the far
// history leaves
// (a slot holds a row of the columns a unit needs in whole groups of 32: at most
// two ranges, one wraps around in x, each with a partial group at an end)
constexpr int SS_GROUPS = SS_THREADS / 32 + 3;
constexpr int SS_COEF_B = 1024, SS_VEC_B = 256;  // bytes of a group: 4 coefficients, one vector
constexpr int SS_GRAM_SLOT = SS_GROUPS * (SS_COEF_B + SS_VEC_B);
constexpr int SS_UPD_SLOT = SS_GROUPS * (SS_COEF_B + SS_VEC_B + 256 + 64);  // the field and the flags too
constexpr int SS_DYN_MAX = 210 * 1024;
__host__ __device__ constexpr int ss_gram_ring(int L) {
    const int fit = (SS_DYN_MAX - ss_nb_bytes(L) - ss_far_bytes(L)) / SS_GRAM_SLOT;
    return fit < 12 ? fit : 12;
}
constexpr int SS_UPD_RING = 9;
constexpr size_t SS_GRAM_DSMEM = SS_DYN_MAX;
constexpr size_t SS_UPD_DSMEM = (size_t)SS_UPD_RING * SS_UPD_SLOT + ss_nb_bytes(SS_MAXL - 1);

// The pending units of a sweep: per system strips times `rows` row ranges, the
// system with more levels first (its units take longest).  A Gram sweep of
// more than SS_ONE levels is two parts, each a march of its own over all
// strips: the sums among p_0 .. p_7, then those with p_8 and up; one thread's
// registers do not hold the windows of so many levels and all their sums.
constexpr int SS_ONE = 8;    // most levels of a Gram sweep in one part
constexpr int SS_SPLIT = 7;  // levels of the first part otherwise
struct SsPlan {
    int first, rows, total;
    int lev[2], parts[2], strips[2], units[2];
    __host__ __device__ __forceinline__ void make(int nx, bool gram, int l0, int l1, int row_ranges) {
        lev[0] = l0;
        lev[1] = l1;
        first = l1 >= l0 ? 1 : 0;
        rows = row_ranges;
        for (int s = 0; s < 2; ++s) {
            parts[s] = gram && lev[s] > SS_ONE ? 2 : 1;
            const int w = SS_THREADS - 2 * (lev[s] < 0 ? 0 : lev[s]);
            strips[s] = (nx + w - 1) / w;
            units[s] = lev[s] < 0 ? 0 : strips[s] * rows * parts[s];
        }
        total = units[0] + units[1];
    }
};

// The unit a block marches, and the copies of one of its rows.
struct SsCopy {
    const void* src;      // of row 0
    unsigned stride;      // bytes from row to row
    unsigned bytes;
    unsigned dst;         // place in the ring slot
    int lag;              // rows behind the step's row
};
struct SsUnit {
    int s, part, n, strip, halo, ya, yb, rst, fin;
    SsCopy copy[8];
    int copies, bytes;    // of a row
    int y0, steps;        // row of step 0 (outside the lattice: negative), steps
    int ring, slots, slot_bytes;  // the ring in use (ss_ring_id)
};
constexpr int SS_RINGS = 2 + SS_MAXL - SS_FAR + 1, SS_RING_MAX = 12;
// A ring per row count, each with its own phases: update sweeps, Gram sweeps
// without and (each level count) with a far history.
__host__ __device__ constexpr int ss_ring_id(int L, bool gram) { return !gram ? 0 : (L < SS_FAR ? 1 : L - SS_FAR + 2); }

struct SsSmem {
    double red[SS_WARPS][SS_NG];  // block reduction of the Gram sums
    unsigned long long full[SS_RINGS][SS_RING_MAX];   // a row's copies have landed
    unsigned long long empty[SS_RINGS][SS_RING_MAX];  // a row has been taken
    int slot[2][SS_RINGS], par[2][SS_RINGS];          // next slot and phase parity: marching side, producer
    SsPlan plan;
    SsUnit u;
    int march;                    // what marches the unit (-1: there is none)
    int go, dead;                 // the producer's order: 1 a unit, 0 end
    double c[2][SS_MAXL + 1];     // update coefficients
};

// The one instance of a block, and its dynamic shared memory.
__device__ __forceinline__ SsSmem& ss_sm() {
    __shared__ SsSmem sm;
    return sm;
}
extern __shared__ __align__(128) unsigned char ss_dyn[];

// Barriers: of the marching threads (and of 256-thread kernels), and of a
// marching block with its producer's warpgroup.
constexpr int SS_BLOCK = SS_THREADS + 128;
__device__ __forceinline__ void ss_sync_march() { asm volatile("bar.sync 1, %0;" ::"n"(SS_THREADS) : "memory"); }
__device__ __forceinline__ void ss_sync_block() { asm volatile("bar.sync 2, %0;" ::"n"(SS_THREADS + 32) : "memory"); }

__device__ __forceinline__ unsigned ss_saddr(const void* p) { return (unsigned)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void ss_bar_arrive(unsigned bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void ss_bar_expect(unsigned bar, unsigned bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool ss_bar_try(unsigned bar, unsigned par) {
    unsigned ok;
    asm volatile(
        "{\n.reg .pred p;\n"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n"
        "selp.u32 %0, 1, 0, p;\n}\n"
        : "=r"(ok) : "r"(bar), "r"(par) : "memory");
    return ok != 0;
}
// Waits for the phase of parity `par`, a bounded number of polls; when they run
// out the solve is marked failed and no later wait of the block polls again.
__device__ __forceinline__ void ss_bar_wait(unsigned bar, unsigned par, int* error) {
    volatile int* dead = &ss_sm().dead;
#pragma unroll 1
    for (int n = 0; !ss_bar_try(bar, par); ++n) {
        if (*dead) return;
        if (n >= (1 << 20)) {
            *dead = 1;
            atomicExch(error, 1);
        }
    }
}
// Bulk copies go through the async proxy: without a fence on the way from one to
// the other they are not ordered after ordinary accesses to the same memory:
// global and shared (what one launch writes and marches), or shared alone (a
// unit's rows where the next unit's ring lies).  The marching threads issue them,
// around the barriers that lead to the producer; in the producer itself, at the
// start of each unit, the fence cost 0.7 us a step at 256x64.
__device__ __forceinline__ void ss_proxy_fence() { asm volatile("fence.proxy.async;" ::: "memory"); }
__device__ __forceinline__ void ss_proxy_fence_shared() { asm volatile("fence.proxy.async.shared::cta;" ::: "memory"); }
__device__ __forceinline__ void ss_bulk(unsigned dst, const void* src, unsigned bytes, unsigned bar) {
    asm volatile("cp.async.bulk.shared::cta.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(dst),
                 "l"(src), "r"(bytes), "r"(bar) : "memory");
}

// Once per launch of a marching kernel, by the whole block.
__device__ __forceinline__ void ss_smem_init() {
    SsSmem& sm = ss_sm();
    const int t = threadIdx.x;
    if (t < 2 * SS_RINGS * SS_RING_MAX) {
        const unsigned bar = ss_saddr(&sm.full[0][0]) + 8u * (unsigned)t;  // full, then empty
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;" ::"r"(bar) : "memory");
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
        asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
    }
    if (t < SS_RINGS) {
        sm.slot[0][t] = sm.slot[1][t] = 0;
        sm.par[0][t] = 0;
        sm.par[1][t] = 1;  // the phase before the first counts as done
    }
    if (t == 0) sm.dead = 0;
    __syncthreads();
}

// The groups of 32 columns a unit's columns [lo, hi) come from, taken
// modulo nx: one range, or two where the unit wraps around.
struct SsCols {
    int g0, n0;  // first range: groups g0 .. g0 + n0 - 1
    int g1, n1;  // second range (n1 = 0: none)
    __device__ __forceinline__ SsCols(int lo, int hi, int nx) {
        g1 = n1 = 0;
        int a = lo, b = hi;
        if (hi - lo >= nx || (lo < 0 && hi > nx)) {
            a = 0;
            b = nx;
        } else if (lo < 0) {
            a = 0;
            g1 = (nx + lo) >> 5;
            n1 = ((nx + 31) >> 5) - g1;
        } else if (hi > nx) {
            b = nx;
            n1 = (hi - nx + 31) >> 5;
        }
        g0 = a >> 5;
        n0 = ((b + 31) >> 5) - g0;
    }
    // position of column x in the ring's row
    __device__ __forceinline__ int pos(int x) const {
        const int g = (x >> 5) - g0;
        return g >= 0 && g < n0 ? x - g0 * 32 : n0 * 32 + x - g1 * 32;
    }
};
__device__ __forceinline__ SsCols ss_cols(const SsArgs& a, const SsUnit& u, int L, int& own_w, int& lo) {
    const int w = SS_THREADS - 2 * u.halo, x0 = u.strip * w;
    own_w = min(w, a.nx - x0);
    lo = x0 - L;
    return SsCols(lo, x0 + own_w + L, a.nx);
}

// The producer's warp: the rows of the placed unit into the ring, in order
// (rows outside the lattice: row 0 / ny - 1, which are solid and therefore
// zero), one copy a lane.
__device__ __forceinline__ void ss_produce(const SsArgs& a) {
    SsSmem& sm = ss_sm();
    const SsUnit& u = sm.u;
    const int lane = threadIdx.x & 31, ring = u.ring, R = u.slots, steps = u.steps, y0 = u.y0;
    int slot = sm.slot[1][ring];
    unsigned par = (unsigned)sm.par[1][ring];
    const bool mine = lane < u.copies;
    const SsCopy q = u.copy[mine ? lane : 0];
    const int bytes = u.bytes, last = a.ny - 1;
    const unsigned base = ss_saddr(ss_dyn) + q.dst;
#pragma unroll 1
    for (int i = 0; i < steps; ++i) {
        ss_bar_wait(ss_saddr(&sm.empty[ring][slot]), par, &a.ctl->error);
        const unsigned bar = ss_saddr(&sm.full[ring][slot]);
        if (lane == 0) ss_bar_expect(bar, (unsigned)bytes);
        __syncwarp();
        if (mine) {
            const int y = min(max(y0 + i - q.lag, 0), last);
            ss_bulk(base + (unsigned)(slot * u.slot_bytes),
                    static_cast<const char*>(q.src) + (unsigned long long)(unsigned)y * q.stride, q.bytes, bar);
        }
        if (++slot == R) { slot = 0; par ^= 1u; }
    }
    __syncwarp();
    if (lane == 0) {
        sm.slot[1][ring] = slot;
        sm.par[1][ring] = (int)par;
    }
}

__device__ __forceinline__ void lds(double& v, unsigned a) { asm volatile("ld.shared.f64 %0, [%1];" : "=d"(v) : "r"(a)); }
__device__ __forceinline__ void lds(float& v, unsigned a) { asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(a)); }
__device__ __forceinline__ void lds(unsigned& v, unsigned a) {  // 16 bits, zero-extended
    asm volatile("{\n.reg .u16 h;\nld.shared.u16 h, [%1];\ncvt.u32.u16 %0, h;\n}" : "=r"(v) : "r"(a));
}
__device__ __forceinline__ void lds2(double& v, double& w, unsigned a) {
    asm volatile("ld.shared.v2.f64 {%0, %1}, [%2];" : "=d"(v), "=d"(w) : "r"(a));
}
__device__ __forceinline__ void sts(unsigned a, double v) { asm volatile("st.shared.f64 [%0], %1;" ::"r"(a), "d"(v) : "memory"); }
__device__ __forceinline__ void sts2(unsigned a, double v, double w) {
    asm volatile("st.shared.v2.f64 [%0], {%1, %2};" ::"r"(a), "d"(v), "d"(w) : "memory");
}

// GRAM: the sums of the products p_k p_j, k <= j, J <= j <= L, over the unit's
// own nodes, left in acc (zero on threads without an own column).
// else: d = sum_{j <= L} c_j p_j at the unit's own nodes, added to the field
// (final; solid-boundary nodes set to 0) or to the correction x.
template <int L, bool GRAM, int J, typename FT, int NA>
__device__ __forceinline__ void ss_march(const SsArgs& a, double (&acc)[NA]) {
    constexpr int NT = SS_THREADS;
    // levels whose row is kept in shared memory until it is complete (level k
    // for L - k steps): those needed longer than the registers' three rows
    constexpr bool FAR = GRAM && L >= SS_FAR;
    constexpr SsFar far(L);
    // circular windows: levels [j][UP], coefficients [U]
    constexpr int U = GRAM && !FAR ? (L + 1 < 3 ? 3 : L + 1) : (L + 3) / 3 * 3;
    constexpr int UP = GRAM && !FAR ? U : 3;
    constexpr int R = GRAM ? ss_gram_ring(L) : SS_UPD_RING, RID = ss_ring_id(L, GRAM);
    constexpr unsigned SLOT = GRAM ? SS_GRAM_SLOT : SS_UPD_SLOT;
    constexpr unsigned OV = SS_GROUPS * SS_COEF_B, OF = OV + SS_GROUPS * SS_VEC_B, OT = OF + SS_GROUPS * 256;
    constexpr int G0 = J * (J + 1) / 2;  // slot of the first sum taken
    SsSmem& sm = ss_sm();
    const int t = threadIdx.x;
    bool own;
    int slot = sm.slot[0][RID];
    unsigned par = (unsigned)sm.par[0][RID];
    unsigned oc, ov, of = 0, ot = 0;
    FT* fout = nullptr;      // this column's field at row ya (update sweep)
    const double* xin = nullptr;
    {
        const SsUnit& u = sm.u;
        int own_w, lo;
        const SsCols cols = ss_cols(a, u, L, own_w, lo);
        own = t >= L && t < L + own_w;
        int xc = lo + min(t, own_w + 2 * L - 1);  // threads past the unit's columns repeat the last one
        xc %= a.nx;
        if (xc < 0) xc += a.nx;
        const int pos = cols.pos(xc);
        oc = (unsigned)((pos >> 5) * SS_COEF_B + (pos & 31) * 8);
        ov = OV + (unsigned)pos * 8;
        if (!GRAM) {
            of = OF + (unsigned)(pos * (int)sizeof(FT));
            ot = OT + (unsigned)(pos * 2);
            const long long n = (long long)u.ya * a.P + xc;
            fout = static_cast<FT*>(a.field[u.s]) + n;
            xin = a.sys[u.s].x + n;
        }
        if (t == 0) {  // the row's copies, for the producer
            SsUnit& v = sm.u;
            int n = 0, bytes = 0;
            auto add = [&](const void* base, int group, unsigned off, int lag) {  // `group` bytes per 32 columns
                for (int r = 0; r < 2; ++r) {
                    const int g = r ? cols.g1 : cols.g0, k = r ? cols.n1 : cols.n0;
                    if (!k) continue;
                    SsCopy& q = v.copy[n++];
                    q.src = static_cast<const char*>(base) + (long long)g * group;
                    q.stride = (unsigned)(a.P >> 5) * (unsigned)group;
                    q.bytes = (unsigned)(k * group);
                    q.dst = off + (unsigned)(r ? cols.n0 * group : 0);
                    q.lag = lag;
                    bytes += k * group;
                }
            };
            if (L > 0) add(a.sys[u.s].coef, SS_COEF_B, 0, 0);
            add(u.rst == 0 ? a.sys[u.s].rhs : a.sys[u.s].r, SS_VEC_B, OV, 0);
            if (!GRAM && u.fin) {
                add(a.field[u.s], 32 * (int)sizeof(FT), OF, L);
                add(a.ntype, 64, OT, L);
            }
            v.copies = n;
            v.bytes = bytes;
            v.y0 = u.ya - L;
            v.steps = u.yb - u.ya + 2 * L;
            v.ring = RID;
            v.slots = R;
            v.slot_bytes = (int)SLOT;
            sm.go = 1;
        }
    }
    const unsigned base = ss_saddr(ss_dyn), full = ss_saddr(&sm.full[RID][0]), empty = ss_saddr(&sm.empty[RID][0]);
    // this thread's place in the neighbour rows ([parity][level pair][column + 1])
    constexpr unsigned NBR = ss_row_bytes(), NBP = NBR * ((L + 1) / 2);
    const unsigned nb = base + R * SLOT + 16u * (unsigned)t;
    const unsigned far_base = base + R * SLOT + 2 * NBP + 8u * (unsigned)t;
#pragma unroll
    for (int j = 0; j < L; j += 2) sts2(nb + 16 + NBP + NBR * (unsigned)(j / 2), 0.0, 0.0);  // read by step 0
    ss_sync_block();  // the producer starts
    const int steps = sm.u.steps;
    const bool fin = !GRAM && sm.u.fin, more = !GRAM && sm.u.rst > 0;
    double Pw[L + 1][UP];
    double cE[U], cW[U], cN[U], cS[U];
    double dsum[L + 1], cf[L + 1];
    double g[NA];
    double nl1 = 0.0, nr1 = 0.0;  // the odd level's neighbours of the last load
#pragma unroll
    for (int j = 0; j <= L; ++j) {
#pragma unroll
        for (int k = 0; k < UP; ++k) Pw[j][k] = 0.0;
        dsum[j] = 0.0;
        cf[j] = GRAM ? 0.0 : sm.c[sm.u.s][j];
    }
#pragma unroll
    for (int k = 0; k < U; ++k) { cE[k] = 0.0; cW[k] = 0.0; cN[k] = 0.0; cS[k] = 0.0; }
#pragma unroll
    for (int k = 0; k < NA; ++k) g[k] = 0.0;
    FT fv = FT(0);
    unsigned ty = 0;
    // the next row's values from the ring (row i + 1's at the end of step i)
    auto take = [&](double& p, double& ce, double& cw, double& cn, double& cs) {
        ss_bar_wait(full + 8u * (unsigned)slot, par, &a.ctl->error);
        const unsigned d = base + (unsigned)slot * SLOT;
        lds(p, d + ov);
        if (L > 0) {
            lds(ce, d + oc);
            lds(cw, d + oc + 256);
            lds(cn, d + oc + 512);
            lds(cs, d + oc + 768);
        }
        if (!GRAM && fin) {
            lds(fv, d + of);
            lds(ty, d + ot);
        }
        if (++slot == R) { slot = 0; par ^= 1u; }
    };
    take(Pw[0][0], cE[0], cW[0], cN[0], cS[0]);
#pragma unroll 1
    for (int b = 0; b < steps; b += U) {
#pragma unroll
        for (int u = 0; u < U; ++u) {
            const int i = b + u;
            if (i >= steps) break;
            const unsigned wr = nb + 16 + ((i & 1) ? NBP : 0u), rd = nb + ((i & 1) ? 0u : NBP);
            double row[L + 1];
            if (FAR && i >= 2 * L) {
#pragma unroll
                for (int k = 0; k + 3 <= L; ++k)
                    lds(row[k], far_base + 8u * NT * (unsigned)(far.ring[k] * U + (u + far.shift[k] + U - (L - k)) % U));
            }
#pragma unroll
            for (int j = 0; j < L; ++j) {
                // level j + 1 at row tau - j - 1 from level j at rows tau - j
                // (this step), tau - j - 1 and its x neighbours (the step
                // before), tau - j - 2 (two before); two levels' neighbours a load
                double l, r;
                if ((j & 1) == 0) {
                    lds2(l, nl1, rd + NBR * (unsigned)(j / 2));
                    lds2(r, nr1, rd + 32 + NBR * (unsigned)(j / 2));
                } else {
                    l = nl1;
                    r = nr1;
                }
                const int c = (u + U - 1 - j) % U;
                // N p in the CSR order of an interior row without its centre: S, W, E, N
                Pw[j + 1][u % UP] = cS[c] * Pw[j][(u + UP - 2) % UP] + cW[c] * l + cE[c] * r + cN[c] * Pw[j][u % UP];
                if ((j & 1) == 1 || j + 1 == L)
                    sts2(wr + NBR * (unsigned)(j / 2), Pw[j & ~1][u % UP], (j & 1) ? Pw[j][u % UP] : 0.0);
            }
            ss_sync_march();  // the neighbours' values of this step; row i taken by all
            if (t == 0) ss_bar_arrive(empty + 8u * (unsigned)(slot == 0 ? R - 1 : slot - 1));
            // what follows needs no other warp
            if (FAR) {
#pragma unroll
                for (int k = 0; k + 3 <= L; ++k)
                    sts(far_base + 8u * NT * (unsigned)(far.ring[k] * U + (u + far.shift[k]) % U), Pw[k][u % UP]);
            }
            const FT f_now = fv;
            const unsigned t_now = ty;
            // row tau - L is complete: p_k from the registers' windows, or from
            // shared memory where it was put L - k steps ago
            if (GRAM) {
#pragma unroll
                for (int k = FAR ? L - 2 : 0; k <= L; ++k) row[k] = Pw[k][(u + 2 * UP - (L - k)) % UP];
            }
            if (i + 1 < steps)
                take(Pw[0][(u + 1) % UP], cE[(u + 1) % U], cW[(u + 1) % U], cN[(u + 1) % U], cS[(u + 1) % U]);
            if (GRAM) {
                if (i >= 2 * L) {
#pragma unroll
                    for (int j = J; j <= L; ++j)
#pragma unroll
                        for (int k = 0; k <= j; ++k) g[GRAM ? ss_gslot(k, j) - G0 : 0] += row[k] * row[j];
                }
            } else {
                // partial sums move one level and one row a step
#pragma unroll
                for (int j = L; j >= 1; --j) dsum[j] = dsum[j - 1] + cf[j] * Pw[j][u % UP];
                dsum[0] = cf[0] * Pw[0][u % UP];
                if (i >= 2 * L) {
                    if (own) {
                        double d = dsum[L];
                        if (more) d += __ldcg(xin);
                        const unsigned ft = t_now;
                        if (!fin) __stcg(const_cast<double*>(xin), d);
                        else if (!(ft & M_SOLID)) *fout = (FT)((double)f_now + d);
                        else if (ft & SOLID_BOUNDARY) *fout = FT(0);
                    }
                    fout += a.P;
                    xin += a.P;
                }
            }
        }
    }
    if (GRAM) {
#pragma unroll
        for (int k = 0; k < NA; ++k) acc[k] = own ? g[k] : 0.0;
    }
    if (t == 0) {
        sm.slot[0][RID] = slot;
        sm.par[0][RID] = (int)par;
    }
    // the last step's readers are done before the next unit writes
    ss_proxy_fence_shared();
    ss_sync_march();
}

// ---- units ------------------------------------------------------------------------
// The sweep's plan and the block's units live in shared memory, not in the
// registers of the code around the marches (whose own allocation they would
// cut).  Starts a sweep; false when it has nothing to march.
__device__ __forceinline__ bool ss_begin(const SsArgs& a, bool gram, int l0, int l1) {
    SsSmem& sm = ss_sm();
    ss_sync_march();
    if (threadIdx.x == 0) sm.plan.make(a.nx, gram, l0, l1, (gram ? a.gram_rows : a.upd_rows)[l0 + 1][l1 + 1]);
    ss_sync_march();
    return sm.plan.total > 0;
}
// Places unit n in shared memory and returns its march: the level count, -1
// when there is no such unit.
__device__ __forceinline__ int ss_take_unit(const SsArgs& a, bool gram, int n) {
    SsSmem& sm = ss_sm();
    if (threadIdx.x == 0) {
        const SsPlan& p = sm.plan;
        int march = -1;
        if (n < p.total) {
            SsUnit& u = sm.u;
            const int s = n < p.units[p.first] ? p.first : 1 - p.first;
            if (s != p.first) n -= p.units[p.first];
            const int per = p.strips[s] * p.rows;
            u.part = p.parts[s] > 1 && n < per ? 1 : 0;  // the larger part first
            if (n >= per) n -= per;
            const int rr = n / p.strips[s];
            u.s = s;
            u.n = n;
            u.strip = n - rr * p.strips[s];
            u.ya = (int)((long long)rr * a.ny / p.rows);
            u.yb = (int)((long long)(rr + 1) * a.ny / p.rows);
            u.halo = p.lev[s];
            u.rst = ldc(&a.ctl->sys[s].rst);
            u.fin = !gram && ldc(&a.ctl->sys[s].bmode) == SS_B_FINAL;
            march = p.parts[s] > 1 && !u.part ? SS_SPLIT : p.lev[s];
        }
        sm.march = march;
    }
    ss_sync_march();
    const int m = sm.march;
    ss_sync_march();
    return m;
}

// Sums of N per-thread values over the warp.  A lane halves the values it
// holds in each of five exchanges (it keeps one half and hands over the
// other), so N values take about N shuffles; put(k, v) gets value k's sum on
// one lane.
template <int N, int OFF, typename F>
__device__ __forceinline__ void ss_warp_sums(const double (&v)[N], int lane, F put) {
    if constexpr (OFF == 0) {
#pragma unroll
        for (int k = 0; k < N; ++k)
            put(k, v[k]);
    } else {
        constexpr int H = (N + 1) / 2;
        const bool up = lane & OFF;
        double h[H];
#pragma unroll
        for (int k = 0; k < H; ++k) {
            const double hi = k + H < N ? v[k + H] : 0.0;
            h[k] = (up ? hi : v[k]) + __shfl_xor_sync(0xffffffffu, up ? v[k] : hi, OFF);
        }
        ss_warp_sums<H, OFF / 2>(h, lane,
                                 [&](int k, double x) { if (!up || k + H < N) put(up ? k + H : k, x); });
    }
}

// A unit's sums of system s.
__device__ __forceinline__ double* ss_part(const SsArgs& a, int s, int unit) {
    return a.part + ((long long)s * a.maxu + unit) * SS_NG;
}

// Sums of N per-thread values over the block into part[0 .. N).
template <int N>
__device__ __forceinline__ void ss_block_sums(const double (&v)[N], double* part) {
    SsSmem& sm = ss_sm();
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    ss_warp_sums<N, 16>(v, lane, [&](int k, double x) { sm.red[warp][k] = x; });
    ss_sync_march();
    for (int k = threadIdx.x; k < N; k += SS_THREADS) {
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < SS_WARPS; ++w) x += sm.red[w][k];
        part[k] = x;
    }
    ss_sync_march();
}

// Sum of n units' first value in a fixed order, one warp, every lane the result.
__device__ __forceinline__ double ss_sum_warp(const double* p, int n) {
    double x = 0.0;
    for (int b = threadIdx.x & 31; b < n; b += 32) x += __ldcg(p + (long long)b * SS_NG);
#pragma unroll
    for (int off = 16; off > 0; off >>= 1) x += __shfl_xor_sync(0xffffffffu, x, off);
    return x;
}

// tot[s][k]: sums over the units, in a fixed order, of both systems' Gram
// entries.  Warp w takes the units w, w + 8, ..; lane l of it the entries
// l, l + 32, l + 64; then the warps' sums are added up.  A chain of waits for
// L2: SS_SUM_U units of both systems are in flight at a time (one warp per
// entry, its lanes across the units, waited for L2 and for a sum over the lanes
// once per entry: 9 to 13 thousand cycles at 45 entries of 70 to 140 units,
// where this takes 2 to 3).
constexpr int SS_SUM_U = 5;
__device__ __forceinline__ void ss_unit_sums(const SsArgs& a, const int (&ng)[2], const int (&n)[2], double (*tot)[SS_NG]) {
    constexpr int C = (SS_NG + 31) / 32;
    double(*red)[2 * SS_NG] = reinterpret_cast<double(*)[2 * SS_NG]>(ss_dyn);  // the march has ended
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    double v[2][C] = {};
    for (int b = warp; b < n[0] || b < n[1]; b += SS_WARPS * SS_SUM_U) {
        double x[SS_SUM_U][2][C];
#pragma unroll
        for (int i = 0; i < SS_SUM_U; ++i)
#pragma unroll
            for (int s = 0; s < 2; ++s)
#pragma unroll
                for (int c = 0; c < C; ++c) {
                    const int u = b + i * SS_WARPS, k = lane + 32 * c;
                    x[i][s][c] = u < n[s] && k < ng[s] ? __ldcg(ss_part(a, s, u) + k) : 0.0;
                }
#pragma unroll
        for (int i = 0; i < SS_SUM_U; ++i)
#pragma unroll
            for (int s = 0; s < 2; ++s)
#pragma unroll
                for (int c = 0; c < C; ++c) v[s][c] += x[i][s][c];
    }
#pragma unroll
    for (int s = 0; s < 2; ++s)
#pragma unroll
        for (int c = 0; c < C; ++c)
            if (lane + 32 * c < ng[s]) red[warp][SS_NG * s + lane + 32 * c] = v[s][c];
    ss_sync_march();
    for (int k = threadIdx.x; k < 2 * SS_NG; k += SS_THREADS) {
        const int s = k / SS_NG, e = k - s * SS_NG;
        if (e >= ng[s]) continue;
        double x = 0.0;
#pragma unroll
        for (int w = 0; w < SS_WARPS; ++w) x += red[w][k];
        tot[s][e] = x;
    }
    ss_proxy_fence_shared();  // bulk copies of a later unit write here
}

// Levels of the Gram sweep of system s (-1: none pending).
__device__ __forceinline__ int ss_gram_levels(const SsArgs& a, int s) {
    const GmresSys* S = &a.ctl->sys[s];
    const int lt = ldc(&S->lto);
    return ldc(&S->active) && lt > 0 ? lt : -1;
}

// One unit of the Gram sweep (the sums with p_J and up), as placed in shared
// memory.
template <int L, int J>
__device__ __forceinline__ void ss_gram_march(const SsArgs& a) {
    constexpr int NG = (L + 1) * (L + 2) / 2 - J * (J + 1) / 2;
    double acc[NG];
    ss_march<L, true, J, float>(a, acc);
    const SsUnit& u = ss_sm().u;
    ss_block_sums<NG>(acc, ss_part(a, u.s, u.n) + J * (J + 1) / 2);
}
// Unit n of the Gram sweep, and of the update sweep.  One unit per block: a
// loop over units around this switch made the compiler keep (and spill)
// registers across the marches, 80 to 300 bytes of local memory a thread and
// step at 7 to 10 levels; without it no march spills.
__device__ __forceinline__ void ss_gram_unit(const SsArgs& a, int n) {
    switch (ss_take_unit(a, true, n)) {
#define KOFM_SS(l, j) \
    case l: ss_gram_march<l, j>(a); break;
        KOFM_SS(1, 0) KOFM_SS(2, 0) KOFM_SS(3, 0) KOFM_SS(4, 0) KOFM_SS(5, 0) KOFM_SS(6, 0)
        KOFM_SS(7, 0) KOFM_SS(8, 0) KOFM_SS(9, SS_SPLIT + 1) KOFM_SS(10, SS_SPLIT + 1)
#undef KOFM_SS
        default: break;
    }
}

// Serial step of a Gram sweep of lev(s) levels (-1: none), run by the last
// block: sums(tot) gets the entries, then per system one warp for the cycle and
// one for the basis's rank.  bytes(s): what the sweep moved, per node.
template <bool ORDERED, typename LEV, typename BYTES, typename SUMS>
__device__ __forceinline__ void ss_gram_serial(const SsArgs& a, LEV lev, BYTES bytes, SUMS sums) {
    __shared__ double tot[2][SS_NG];
    __shared__ GmresSys sS[2];
    __shared__ SsCycleSmem cs[2];
    const int warp = threadIdx.x >> 5;
    SsSysWord w[2];
#pragma unroll
    for (int s = 0; s < 2; ++s) w[s].load(a.ctl, s);
    sums(tot);
    for (int s = 0; s < 2; ++s) w[s].put(sS[s]);
    ss_sync_march();
    const int s = warp & 1, L = lev(s);
    if (L > 0) {
        if (threadIdx.x == 32 * s) sS[s].abytes += bytes(s);
        ss_gram_begin(a, sS[s], tot[s], L, cs[s]);
    }
    ss_sync_march();
    SsCycle c;
    if (L > 0 && sS[s].active) {
        if (warp < 2) ss_cycle<ORDERED>(c, cs[s], L, a.K, a.rel_tol, sS[s].rinv);
        else if (warp < 4) ss_rank(cs[s], L + 1);
    }
    ss_sync_march();
    if (warp < 2 && L > 0 && sS[s].active) ss_gram_end(a, sS[s], s, L, cs[s], c);
    ss_sync_march();
    for (int q = 0; q < 2; ++q)
        if (lev(q) > 0) sp_sys_store(a.ctl, q, sS[q]);
    if (threadIdx.x == 0) {
        trace_barrier(a.ctl);
        __stcg(&a.ctl->passes, ldc(&a.ctl->passes) + 1);
        __stcg(&a.ctl->any_active, (int)(sS[0].active || sS[1].active));
    }
}
// After a march: the sums over the units in a fixed order.
__device__ __forceinline__ void ss_gram_serial(const SsArgs& a) {
    const SsPlan& pl = ss_sm().plan;
    ss_gram_serial<false>(
        a, [&](int s) { return pl.lev[s]; },
        [&](int s) { return 40.0 * pl.parts[s]; },  // p_0 and the coefficients
        [&](double (*tot)[SS_NG]) {
            int ng[2], n[2];
#pragma unroll
            for (int s = 0; s < 2; ++s) {
                ng[s] = pl.lev[s] > 0 ? (pl.lev[s] + 1) * (pl.lev[s] + 2) / 2 : 0;
                n[s] = ng[s] ? pl.strips[s] * pl.rows : 0;
            }
            ss_unit_sums(a, ng, n, tot);
        });
}

// Levels of the update sweep of system s (-1: nothing for a march to do).
__device__ __forceinline__ int ss_upd_levels(const SsArgs& a, int s) {
    const GmresSys* S = &a.ctl->sys[s];
    const int m = ldc(&S->bmode), kk = ldc(&S->kk);
    if (m != SS_B_FINAL && m != SS_B_UPDATE) return -1;
    // (two levels run as three, the third with coefficient 0: the compiler keeps
    // the march of two in local memory, at 1.4 times the time)
    return kk <= 1 ? 0 : (kk == 3 ? 3 : kk - 1);
}

template <typename FT>
__device__ __forceinline__ void ss_upd_unit(const SsArgs& a, int n) {
    if (threadIdx.x < 2 * (SS_MAXL + 1)) {  // (read after the barriers of ss_take_unit)
        const int s = threadIdx.x / (SS_MAXL + 1), i = threadIdx.x % (SS_MAXL + 1);
        ss_sm().c[s][i] = i < SS_MAXL ? ldc(&a.ctl->sys[s].h[i]) : 0.0;
    }
    double none[1];
    switch (ss_take_unit(a, false, n)) {
#define KOFM_SS(l) \
    case l: ss_march<l, false, 0, FT>(a, none); break;
        KOFM_SS(0) KOFM_SS(1) KOFM_SS(3) KOFM_SS(4) KOFM_SS(5)
        KOFM_SS(6) KOFM_SS(7) KOFM_SS(8) KOFM_SS(9)
#undef KOFM_SS
        default: break;
    }
}

// field += x on fluid nodes and 0 on solid-boundary nodes of a system whose
// solve ended at a convergence test (pointwise); a solve that met a NaN
// residual, or ran no cycle, leaves its fluid nodes as they were.
template <typename FT>
__device__ __forceinline__ void ss_write_units(const SsArgs& a) {
    const int cpr = (a.P / 2 + SS_THREADS - 1) / SS_THREADS;
    const int units = a.ny * cpr;
    for (int s = 0; s < 2; ++s) {
        if (ldc(&a.ctl->sys[s].bmode) != SS_B_WRITE) continue;
        const bool has_x = ldc(&a.ctl->sys[s].cycles) > 0 && !ldc(&a.ctl->sys[s].nan);
        FT* f = static_cast<FT*>(a.field[s]);
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            const int y = u / cpr;
            const int x = ((u - y * cpr) * SS_THREADS + threadIdx.x) * 2;
            if (x >= a.nx) continue;
            const long long g = (long long)y * a.P + x;
            const unsigned int t2 = *reinterpret_cast<const unsigned int*>(a.ntype + g);
            const int tt[2] = {(int)(t2 & 0xffff), (int)(t2 >> 16)};
            const double2 xv = has_x ? __ldcg(reinterpret_cast<const double2*>(a.sys[s].x + g)) : make_double2(0.0, 0.0);
            const double dv[2] = {xv.x, xv.y};
            for (int j = 0; j < 2; ++j) {
                if (x + j >= a.nx) continue;
                if (!(tt[j] & M_SOLID)) f[g + j] = (FT)((double)f[g + j] + dv[j]);
                else if (tt[j] & SOLID_BOUNDARY) f[g + j] = FT(0);
            }
        }
    }
}

// End of the update sweep (one thread, every unit done): a kept correction
// waits for its residual sweep, a written field is done.
__device__ __forceinline__ void ss_upd_serial(const SsArgs& a) {
    for (int s = 0; s < 2; ++s) {
        GmresSys* S = &a.ctl->sys[s];
        const int m = ldc(&S->bmode);
        if (m == SS_B_UPDATE) __stcg(&S->ready, 1);
        else if (m != SS_B_NONE) __stcg(&S->written, 1);
        __stcg(&S->bmode, (int)SS_B_NONE);
    }
    __stcg(&a.ctl->passes, ldc(&a.ctl->passes) + 1);
}

// r = b' - A x and ||r||^2 of every system whose cycle kept its correction;
// partial sums in slot 0 of each system, one per block.
__device__ __forceinline__ bool ss_resid_units(const SsArgs& a, const bool act[2]) {
    // units of (row, chunk of 2 x 256 columns): one 32-bit division per unit
    const int cpr = (a.P / 2 + SS_THREADS - 1) / SS_THREADS;
    const int units = a.ny * cpr;
    for (int s = 0; s < 2; ++s) {
        if (!act[s]) continue;
        double acc[1] = {0.0};
        const KoSystem& S = a.sys[s];
        for (int u = blockIdx.x; u < units; u += gridDim.x) {
            const int y = u / cpr;
            const int x = ((u - y * cpr) * SS_THREADS + threadIdx.x) * 2;
            if (x >= a.P) continue;
            const long long g = (long long)y * a.P + x;
            double rr[2] = {0.0, 0.0};
            const long long row = (long long)y * a.P;
#pragma unroll
            for (int j = 0; j < 2; ++j) {
                const int xj = x + j;
                if (xj >= a.nx) continue;
                const long long gj = g + j;
                const int xw = xj > 0 ? xj - 1 : a.nx - 1;
                const int xe = xj + 1 < a.nx ? xj + 1 : 0;
                const double* cf = S.coef + ilv(4, 0, gj);
                // rows 0 and ny-1 are solid: their off-diagonals are 0
                const double dS = y > 0 ? __ldcg(S.x + gj - a.P) : 0.0;
                const double dN = y + 1 < a.ny ? __ldcg(S.x + gj + a.P) : 0.0;
                // CSR order of an interior row: S, W, C, E, N
                // (the rows are not read-only where one launch runs several
                // sub-steps: no non-coherent loads)
                const double Ad = __ldcg(cf + 96) * dS + __ldcg(cf + 32) * __ldcg(S.x + row + xw) + __ldcg(S.x + gj) +
                                  __ldcg(cf) * __ldcg(S.x + row + xe) + __ldcg(cf + 64) * dN;
                rr[j] = __ldcg(S.rhs + gj) - Ad;
            }
            __stcg(reinterpret_cast<double2*>(S.r + g), make_double2(rr[0], rr[1]));
            acc[0] += rr[0] * rr[0] + rr[1] * rr[1];
        }
        ss_block_sums<1>(acc, ss_part(a, s, blockIdx.x));
    }
    return act[0] || act[1];
}

__device__ __forceinline__ void ss_resid_serial(const SsArgs& a, const bool act[2]) {
    __shared__ double tot[2];
    __shared__ GmresSys sS[2];
    sp_sys_load(a.ctl, 0, sS[0]);
    sp_sys_load(a.ctl, 1, sS[1]);
    const int warp = threadIdx.x >> 5;
    if (warp < 2 && act[warp]) {
        const double v = ss_sum_warp(ss_part(a, warp, 0), gridDim.x);
        if ((threadIdx.x & 31) == 0) tot[warp] = v;
    }
    ss_sync_march();
    if (threadIdx.x < 2 && act[threadIdx.x]) ss_resid_step(a, sS[threadIdx.x], threadIdx.x, tot[threadIdx.x]);
    ss_sync_march();
    for (int s = 0; s < 2; ++s)
        if (act[s]) sp_sys_store(a.ctl, s, sS[s]);
    if (threadIdx.x == 0) {
        trace_barrier(a.ctl);
        __stcg(&a.ctl->passes, ldc(&a.ctl->passes) + 1);
        __stcg(&a.ctl->any_active, (int)(sS[0].active || sS[1].active));
    }
}

// Systems whose kept correction waits for its residual.
__device__ __forceinline__ void ss_resid_pending(const SsArgs& a, bool act[2]) {
    for (int s = 0; s < 2; ++s) act[s] = ldc(&a.ctl->sys[s].active) && ldc(&a.ctl->sys[s].ready);
}

// ---- the solver in one cooperative launch --------------------------------------------
// The sweeps above with bounded grid barriers between them; the last block to
// reach a barrier runs the serial step (the same protocol as the
// one-vector-per-sweep solver's).  What a block wrote before the barrier, others
// march after it: so the proxy fences on both sides.
template <typename F>
__device__ __forceinline__ bool ss_sync(const SsArgs& a, F serial) {
    __shared__ int s_last;
    __shared__ unsigned int s_gen;
    const unsigned nblocks = gridDim.x;
    ss_proxy_fence();
    __threadfence();
    ss_sync_march();
    if (threadIdx.x == 0) {
        __threadfence();
        s_gen = ld_acquire_u32(&a.bar->gen);
        const unsigned int ticket = atomicAdd(&a.bar->count, 1u);
        s_last = (ticket == nblocks - 1u);
    }
    ss_sync_march();
    if (s_last) {
        __threadfence();
        serial();
        __threadfence();
        ss_sync_march();
        if (threadIdx.x == 0) {
            atomicExch(&a.bar->count, 0u);
            __threadfence();
            atomicAdd(&a.bar->gen, 1u);
        }
    } else if (threadIdx.x == 0) {
        long long it = 0;
        while (ld_acquire_u32(&a.bar->gen) == s_gen) {
            if (++it > a.spin_limit || ldc(&a.ctl->error)) {
                atomicExch(&a.ctl->error, 1);
                break;
            }
            __nanosleep(100);
        }
    }
    ss_sync_march();
    ss_proxy_fence();
    return ldc(&a.ctl->error) == 0;
}

static_assert(SS_UPD_DSMEM <= SS_GRAM_DSMEM, "the cooperative form's dynamic shared memory");

// A marching kernel's block: its third warpgroup gives its registers to the
// other two and keeps one warp, which fetches the rows of every unit they
// place until told to end; the other two run `body`.
template <typename F>
__device__ __forceinline__ void ss_specialise(const SsArgs& a, F body) {
    ss_smem_init();
    if (threadIdx.x >= SS_THREADS) {
        asm volatile("setmaxnreg.dec.sync.aligned.u32 24;");
        if (threadIdx.x < SS_THREADS + 32) {
            while (true) {
                ss_sync_block();
                if (!*(volatile int*)&ss_sm().go) break;
                ss_produce(a);
            }
        }
        return;
    }
    asm volatile("setmaxnreg.inc.sync.aligned.u32 240;");
    body();
    ss_sync_march();
    if (threadIdx.x == 0) ss_sm().go = 0;
    ss_sync_block();
    // After a wait that ran out, copies may be in flight into this block's shared
    // memory: it stays for a while (1 ms, far above a copy's time) before it ends.
    if (*(volatile int*)&ss_sm().dead)
        for (int i = 0; i < 1000; ++i) __nanosleep(1000);
}

// (returns the rounds run)
template <typename FT>
__device__ __forceinline__ int ss_solve(const SsArgs& a) {
    if (blockIdx.x == 0 && threadIdx.x == 0) __stcg(&a.ctl->t_start, globaltimer_ns());
    // every restart takes at most two rounds (its first and one extension)
    int round = 0;
    while (round < 2 * a.max_restarts + 2) {
        ++round;
        {
            bool act[2];
            ss_resid_pending(a, act);
            if (ss_resid_units(a, act) && !ss_sync(a, [&] { ss_resid_serial(a, act); })) return round;
        }
        {
            if (ss_begin(a, true, ss_gram_levels(a, 0), ss_gram_levels(a, 1))) {
                for (int n = blockIdx.x; n < ss_sm().plan.total; n += gridDim.x) ss_gram_unit(a, n);
                if (!ss_sync(a, [&] { ss_gram_serial(a); })) return round;
            }
        }
        {
            if (ss_begin(a, false, ss_upd_levels(a, 0), ss_upd_levels(a, 1)))
                for (int n = blockIdx.x; n < ss_sm().plan.total; n += gridDim.x) ss_upd_unit<FT>(a, n);
            ss_write_units<FT>(a);
        }
        if (!ldc(&a.ctl->any_active)) return round;
        if (!ss_sync(a, [&] { if (threadIdx.x == 0) ss_upd_serial(a); })) return round;
    }
    return round;
}

template <typename FT>
__global__ void __launch_bounds__(SS_BLOCK, 1)
sstep_kernel(const __grid_constant__ SsArgs a) {
    ss_specialise(a, [&] { ss_solve<FT>(a); });
}

// ---- the same solver as separate sweep launches -----------------------------------------
// Each sweep is its own launch and reads what it has to do from the control
// block: a residual sweep for corrections that were kept, the Gram sweep of
// the pending cycles, the update sweep.  The serial steps run in the last
// block to finish a sweep (ticket counter, no grid barrier and no spin-wait).
// A typical solve is one Gram and one update sweep for both systems.

// True in every thread of the block that finishes a sweep last; that block
// then sees every other block's partial sums.  Resets the ticket counter for
// the next sweep on the stream.
__device__ __forceinline__ bool sp_last_block(const SsArgs& a) {
    __shared__ int s_last;
    __threadfence();
    ss_sync_march();
    if (threadIdx.x == 0) {
        const unsigned int ticket = atomicAdd(&a.queue->count, 1u);
        s_last = ticket == gridDim.x - 1u;
        if (s_last) atomicExch(&a.queue->count, 0u);
    }
    ss_sync_march();
    if (s_last) __threadfence();
    return s_last;
}

// Sub-stepping state of one context (device memory; the host pushes a reset
// when a state is loaded and reads it back when it synchronises).
struct KoStepState {
    double dt;             // kOmega::timeStep
    int steps_per_lb;      // kOmega::stepsPerLB
    int time_since_change; // kOmega::timeSinceTimeStepChange
    int cur;               // sub-step of the running update
    int status;            // KOFM_OK, or the error that stopped updates (sticky until a reset)
    int fail_solves;       // kofm_debug_fail_solves: solves still to report a NaN
    int fail_mask;
    int substeps;          // solves of the last update
    int launches;          // kernel launches of the last update
    int fresh;             // 1: the next sub-step is an update's first (doubling test not yet applied)
    int again;             // 1: the running solve needs another round (no assembly)
    int go;                // 1: the running update is not finished
    long long updates;     // updates run since the last reset
    long long launches_total;  // kernel launches of all updates since the last reset
};

// Control block of a solve: both systems iterating, restart 0, first sweep of
// l0 / l1 levels, a pending failure injection (kofm_debug_fail_solves).
// (MARCH: by the marching threads of a block whose grid is at its barriers)
template <bool MARCH>
__device__ __forceinline__ void ss_ctl_init(GmresControl* ctl, GridBarrier* bar, SsQueue* queue, KoStepState* st,
                                            int l0, int l1) {
    constexpr int NW = (int)(sizeof(GmresControl) / sizeof(unsigned int));
    unsigned int* w = reinterpret_cast<unsigned int*>(ctl);
    const int threads = MARCH ? SS_THREADS : (int)blockDim.x;
    for (int i = threadIdx.x; i < NW; i += threads) w[i] = 0u;
    if (MARCH) ss_sync_march();
    else __syncthreads();
    if (threadIdx.x == 0) {
        int inject = 0;
        if (st->fail_solves > 0) {
            inject = st->fail_mask;
            st->fail_solves--;
        }
        for (int s = 0; s < 2; ++s) {
            ctl->sys[s].active = 1;
            ctl->sys[s].inject = (inject >> s) & 1;
            ctl->sys[s].lto = s == 0 ? l0 : l1;
        }
        ctl->any_active = 1;
        ctl->t_start = globaltimer_ns();
        if (!MARCH) {
            bar->count = 0u;
            bar->gen = 0u;
            queue->count = 0u;
        }
    }
}

__global__ void sp_init_kernel(GmresControl* ctl, GridBarrier* bar, SsQueue* queue, KoStepState* st, int l0, int l1) {
    ss_ctl_init<false>(ctl, bar, queue, st, l0, l1);
}

// (st: the sub-stepping state of the update graph, whose sweeps do nothing once
// an update has stopped with an error; null in the host-driven form)
__device__ __forceinline__ bool sp_stopped(const KoStepState* st) { return st && ldc(&st->status) != 0; }
// A sweep of a further round of the update graph has something to do while the
// round before asked for it.
__device__ __forceinline__ bool sp_idle(const KoStepState* st, int further) {
    return sp_stopped(st) || (further && !ldc(&st->again));
}

__global__ void __launch_bounds__(SS_THREADS)
sp_resid_kernel(const __grid_constant__ SsArgs a, const KoStepState* st, int further) {
    bool act[2];
    if (sp_idle(st, further)) return;
    ss_resid_pending(a, act);
    if (!ss_resid_units(a, act)) return;
    if (sp_last_block(a)) ss_resid_serial(a, act);
}

__global__ void __launch_bounds__(SS_BLOCK, 1)
sp_gram_kernel(const __grid_constant__ SsArgs a, const KoStepState* st, int further) {
    if (sp_idle(st, further)) return;
    ss_specialise(a, [&] {
        if (!ss_begin(a, true, ss_gram_levels(a, 0), ss_gram_levels(a, 1))) return;
        ss_gram_unit(a, blockIdx.x);
        if (sp_last_block(a)) ss_gram_serial(a);
    });
}

// ---- the first Gram sums of a loaded state ------------------------------------------------
// What ends a cycle is rounding (in exact arithmetic |xi_k| stays below rho): a
// last digit of a Gram sum decides whether it ends a vector sooner, at a residual
// of about 1e-6 or of 1e-9 ||b'||.  In a running channel neither shows.  In the
// first solve after kofm_set_state it can: beside a curved wall that passes a
// node at 1e-4, omega starts at 6 nu / (0.075 d^2) and is 1000 at most afterwards,
// ||b'|| is 1e5 to 1e7, and 1e-6 of it is percents of the omega a node further,
// which later steps do not take back.  So that solve takes its sums in one fixed
// order, whatever the form, the row ranges and the units of a march: the nodes in
// so_ranges(L) ranges of whole 32-column groups, a thread every 256th node of a
// range, then the threads of a warp, the warps, the ranges.  It takes all K powers,
// whatever the solves of an earlier state took, and its cycle the reference's
// formulas to the letter (ss_cycle<true>).  Measured on 242
// channels with wavy walls, the fields after 6 steps: with the marches' sums 17
// differ by over 0.8% of omega or k at a node from the fixed order's, by up to
// 60%; with these sums the largest difference is 5e-6 (1e-7 the median).
//
// The powers are formed one after the other in memory and summed in a pass of
// their own: a loaded state's first step takes 80 us more at 256x64, 350 at
// 4096x512 and 2600 at 16384x1024, so only states that need it take it
// (k_first_ordered).  Where the memory for the powers cannot be had, the first
// solve marches like the others.
__host__ __device__ constexpr int so_ranges(int L) { return 148 * (L >= 9 ? 1 : L >= 6 || L == 1 ? 2 : 3); }
constexpr int SO_MAX_RANGES = 148 * 3;

// p_{j+1} = N p_j of both systems.
__global__ void __launch_bounds__(SS_THREADS) sp_power_kernel(const __grid_constant__ SsArgs a, const KoStepState* st, int j) {
    if (sp_stopped(st)) return;
    const int x = blockIdx.x * SS_THREADS + threadIdx.x;
    if (x >= a.nx) return;
    const int xw = x > 0 ? x - 1 : a.nx - 1, xe = x + 1 < a.nx ? x + 1 : 0;
    const KoSystem& S = a.sys[blockIdx.z];
    const double* p = j == 0 ? S.rhs : S.V + (j - 1) * a.D;
    double* out = S.V + j * a.D;
    for (int y = blockIdx.y; y < a.ny; y += gridDim.y) {
        const long long row = (long long)y * a.P, g = row + x;
        const double* cf = S.coef + ilv(4, 0, g);
        // rows 0 and ny - 1 are solid: their off-diagonals are 0
        const double pS = y > 0 ? p[g - a.P] : 0.0, pN = y + 1 < a.ny ? p[g + a.P] : 0.0;
        // (the roundings are part of the result here, so they are written out)
        out[g] = __fma_rn(cf[64], pN, __fma_rn(cf[0], p[row + xe], __fma_rn(cf[96], pS, __dmul_rn(cf[32], p[row + xw]))));
    }
}

// The sums of a range and, in the last block, the serial step; in place of the
// Gram sweep.  Block b: range b of omega, then of k.
__global__ void __launch_bounds__(SS_THREADS, 1)
sp_first_gram_kernel(const __grid_constant__ SsArgs a, const KoStepState* st) {
    __shared__ double red[SS_WARPS][SS_NG];
    if (sp_stopped(st)) return;
    const int lev[2] = {ss_gram_levels(a, 0), ss_gram_levels(a, 1)};
    if (lev[0] < 0 && lev[1] < 0) return;
    // [slot][range] of each system
    double* const part[2] = {a.part, a.part + (long long)SS_NG * SO_MAX_RANGES};
    const int sys = blockIdx.x >= SO_MAX_RANGES, r = blockIdx.x - sys * SO_MAX_RANGES, L = lev[sys];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (L > 0 && r < so_ranges(L)) {
        const int ranges = so_ranges(L);
        const double* const p0 = a.sys[sys].rhs;
        const double* const V = a.sys[sys].V;
        const long long n32 = a.D / 32, g1 = n32 * (r + 1) / ranges * 32;
        double s[SS_NG], p[SS_MAXL + 1];
#pragma unroll
        for (int i = 0; i < SS_NG; ++i) s[i] = 0.0;
        auto load = [&](long long g) {
#pragma unroll
            for (int j = 0; j <= SS_MAXL; ++j) p[j] = j <= L && g < g1 ? __ldcg(j == 0 ? p0 + g : V + (j - 1) * a.D + g) : 0.0;
        };
        long long g = n32 * r / ranges * 32 + threadIdx.x;
        load(g);
        for (; g < g1; g += SS_THREADS) {
            double q[SS_MAXL + 1];
#pragma unroll
            for (int j = 0; j <= SS_MAXL; ++j) q[j] = p[j];
            load(g + SS_THREADS);
#pragma unroll
            for (int j = 0; j <= SS_MAXL; ++j)
#pragma unroll
                for (int i = 0; i <= j; ++i) s[ss_gslot(i, j)] = __fma_rn(q[i], q[j], s[ss_gslot(i, j)]);
        }
#pragma unroll
        for (int i = 0; i < SS_NG; ++i) {
            double x = s[i];
#pragma unroll
            for (int off = 16; off > 0; off >>= 1) x += __shfl_down_sync(0xffffffffu, x, off);
            if (lane == 0) red[warp][i] = x;
        }
        ss_sync_march();
        for (int i = threadIdx.x; i < SS_NG; i += SS_THREADS) {
            double x = 0.0;
#pragma unroll
            for (int w = 0; w < SS_WARPS; ++w) x += red[w][i];
            __stcg(part[sys] + (long long)i * ranges + r, x);
        }
    }
    if (!sp_last_block(a)) return;
    ss_gram_serial<true>(
        a, [&](int s) { return s ? lev[1] : lev[0]; },
        // a power: one and four coefficients in, one out; the sums: all in
        [&](int s) { return 56.0 * (s ? lev[1] : lev[0]) + 8.0; },
        [&](double (*tot)[SS_NG]) {
#pragma unroll
            for (int s = 0; s < 2; ++s)
                for (int i = warp; lev[s] > 0 && i < (lev[s] + 1) * (lev[s] + 2) / 2; i += SS_WARPS) {
                    const double v = sum_slot_warp(part[s], so_ranges(lev[s]), i);
                    if (lane == 0) tot[s][i] = v;
                }
        });
}

// ---- the update on the device -------------------------------------------------------------
// kOmega::Solve (kOmega.cpp:31-73: the doubling test, then sub-steps of
// assembly + both solves, halving dt on a NaN residual) as four launches:
// assembly, Gram sweep, update sweep, and a cooperative kernel for whatever
// the first three did not finish: cycles that asked for more powers, restarts,
// sub-steps.  A usual step has nothing left, and that kernel returns at once;
// so a time step needs neither a host round trip nor a conditional graph node
// (a WHILE node around the same kernels cost 8 to 10 us a step, and a launch
// for a residual sweep that has nothing to do 2).  The update sweep's last
// block takes the decisions of a round; the loop is bounded by counters: a
// solve by its round cap, an update by the halving cap (steps_per_lb <= 2^20)
// and a total of KU_MAX_SUBSTEPS solves.

constexpr int KU_MAX_SUBSTEPS = (1 << 21) + 64;  // above any sequence the halving cap allows

__global__ void ku_reset_kernel(KoStepState* st, double dt, int steps_per_lb) {
    if (threadIdx.x) return;
    st->dt = dt;
    st->steps_per_lb = steps_per_lb;
    st->time_since_change = 0;
    st->cur = 0;
    st->status = 0;
    st->substeps = 0;
    st->launches = 0;
    st->fresh = 1;
    st->again = 0;
    st->go = 0;
    st->updates = 0;
    st->launches_total = 0;
}

__global__ void ku_fail_kernel(KoStepState* st, int n, int mask) {
    if (threadIdx.x) return;
    st->fail_solves = n;
    st->fail_mask = mask;
}

// doubleTimeStep (kOmega.cpp:401-414) as the start of an update applies it
__host__ __device__ __forceinline__ bool ku_doubles(int time_since_change, int steps_per_lb) {
    return time_since_change + 1 >= 20 && steps_per_lb != 1;
}
// Time step of the assembly about to run.
__device__ __forceinline__ double ku_dt(const KoStepState* st) {
    const double dt = ldc(&st->dt);
    return ldc(&st->fresh) && ku_doubles(ldc(&st->time_since_change), ldc(&st->steps_per_lb)) ? dt * 2.0 : dt;
}

// The assembly of an update's first sub-step, and the control block of its
// solve (written by the first block; the sweeps that read it are later
// launches).
template <typename FT>
__global__ void __launch_bounds__(KM_WARPS * 32, KOFM_ASM_MINBLOCKS)
ku_assemble_kernel(const AsmParams p, GmresControl* ctl, GridBarrier* bar, SsQueue* queue, KoStepState* st,
                   const int* lhint, int K) {
    if (ldc(&st->status)) return;
    if (blockIdx.x == 0)
        ss_ctl_init<false>(ctl, bar, queue, st, ss_hint_levels(__ldcg(lhint), K), ss_hint_levels(__ldcg(lhint + 1), K));
    km_assemble<FT>(p, ku_dt(st), blockIdx.x * KM_WARPS + (threadIdx.x >> 5));
}

constexpr int KU_LAUNCHES = 4;  // assembly, Gram and update sweep, the rest; three per further round
// Rounds of a solve that the update enqueues as sweeps of their own after the
// first, before the kernel for the rest: those that the options make usual.  A
// cycle ends at 1e-6 to 1e-9 of its start, so below that a second one follows, of
// few vectors each several; at the default tolerance there is none, and three
// launches with nothing to do would be 6 us.  The rest kernel has one block per SM
// and a barrier's wait between sweeps, which a small lattice does not feel.  With
// rounds left to it and enqueued, us a step at 1e-9, 10 vectors a cycle (one
// round): 256x64 113 and 119, 1001x253 203 and 186, 4096x512 1054 and 893,
// 16384x1024 7190 and 5710; 3 vectors (three rounds): 256x64 94 and 116, 2048x256
// 223 and 231, 4096x512 682 and 665, 16384x1024 5280 and 4870.
__host__ inline int ku_further_rounds(double rel_tol, int K, long long nodes) {
    if (rel_tol >= 1.0e-6 && K >= 3) return 0;
    if (K >= 8) return nodes >= 1 << 17 ? 1 : 0;
    return nodes >= 1 << 20 ? 3 : 0;
}

// Decisions after `rounds` rounds of a solve (one thread): what is left of the
// update.
__device__ __forceinline__ void ku_round_end(const SsArgs& a, KoStepState* st, int rounds, int max_rounds) {
    GmresControl* ctl = a.ctl;
    if (st->fresh) {
        if (ku_doubles(st->time_since_change, st->steps_per_lb)) {
            st->steps_per_lb /= 2;
            st->dt *= 2.0;
        }
        st->time_since_change = st->time_since_change + 1 >= 20 ? 0 : st->time_since_change + 1;
        st->cur = 0;
        st->substeps = 0;
        st->launches = a.launches;
        st->launches_total += a.launches;
        st->updates++;
        st->fresh = 0;
    }
    st->again = 0;
    const int r = ldc(&ctl->rounds) + rounds;
    __stcg(&ctl->rounds, r);
    bool go = false;
    if (ldc(&ctl->error)) {
        st->status = KOFM_ERR_TIMEOUT;
    } else if (ldc(&ctl->sys[0].active) || ldc(&ctl->sys[1].active)) {
        if (r >= max_rounds) st->status = KOFM_ERR_STATE;
        else {
            st->again = 1;
            go = true;
        }
    } else {
        // end of a sub-step: halveTimeStep on a NaN residual (omega first, then
        // k; kOmega.cpp:68-70, 387-399)
        st->substeps++;
        for (int s = 0; s < 2; ++s) {
            if (ldc(&ctl->sys[s].nan)) {
                st->steps_per_lb *= 2;
                st->dt /= 2.0;
                st->cur = 0;
                st->time_since_change = 0;
            }
        }
        if (st->steps_per_lb > (1 << 20) || st->substeps >= KU_MAX_SUBSTEPS) {
            st->status = KOFM_ERR_NAN;  // runaway halving
        } else {
            st->cur++;
            go = st->cur < st->steps_per_lb;
        }
    }
    if (!go) st->fresh = 1;
    st->go = go;
}

// The update sweep.
template <typename FT>
__global__ void __launch_bounds__(SS_BLOCK, 1)
sp_update_kernel(const __grid_constant__ SsArgs a, KoStepState* st, int max_rounds, int further) {
    if (sp_idle(st, further)) return;
    ss_specialise(a, [&] {
        if (ss_begin(a, false, ss_upd_levels(a, 0), ss_upd_levels(a, 1))) ss_upd_unit<FT>(a, blockIdx.x);
        ss_write_units<FT>(a);
        if (sp_last_block(a) && threadIdx.x == 0) {
            ss_upd_serial(a);
            if (st) ku_round_end(a, st, 1, max_rounds);
        }
    });
}

// What is left of an update (cooperative; returns at once where nothing is).
template <typename FT>
__global__ void __launch_bounds__(SS_BLOCK, 1)
ku_rest_kernel(const __grid_constant__ SsArgs a, const __grid_constant__ AsmParams p, KoStepState* st, int max_rounds) {
    if (sp_stopped(st) || !ldc(&st->go)) return;
    ss_specialise(a, [&] {
        // warps whose row rings of the assembly fit in the march's shared memory
        constexpr int AW = (int)(SS_GRAM_DSMEM / km_ring_bytes<FT>()) < SS_WARPS ? (int)(SS_GRAM_DSMEM / km_ring_bytes<FT>())
                                                                               : SS_WARPS;
        while (true) {
            if (!ldc(&st->again)) {
                if (blockIdx.x == 0)
                    ss_ctl_init<true>(a.ctl, a.bar, a.queue, st, ss_hint_levels(__ldcg(a.lhint), a.K),
                                      ss_hint_levels(__ldcg(a.lhint + 1), a.K));
                const int warp = threadIdx.x >> 5, warps = km_warps(p);
                if (warp < AW)
                    for (int w = blockIdx.x * AW + warp; w < warps; w += gridDim.x * AW) km_assemble<FT>(p, ku_dt(st), w);
                if (!ss_sync(a, [] {})) break;
            }
            const int rounds = ss_solve<FT>(a);
            if (!ss_sync(a, [&] { if (threadIdx.x == 0) ku_round_end(a, st, rounds, max_rounds); })) break;
            if (!ldc(&st->go)) return;
        }
        if (threadIdx.x == 0) {  // a barrier's wait ran out
            st->status = KOFM_ERR_TIMEOUT;
            st->go = 0;
        }
    });
}

}  // namespace kofm
