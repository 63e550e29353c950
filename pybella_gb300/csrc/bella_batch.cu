// bella_batch.cu -- the elliptic solves of an ensemble of 2D members with
// uneven grids in one persistent launch (sm_103a).
//
// Every member is the reference's solve (second_projection.py:205-230):
// scipy's BiCGStab on the Jacobi-scaled 9-point system, x0 = 0, stop at
// ||r|| <= max(tol*||b||, atol) with the scipy 1.7 legacy exit ||b|| <= tol.
// Arithmetic: FP64, or double-float on the FP32 pipe (the default: GB300's
// FP64 pipe bounds the FP64 kernel); a double-float member whose FP64 true
// residual misses the tolerance is refined (FP64 residual, batched correction
// solve, FP64 update) by the host driver.
// Each member's operator and Krylov vectors live in its own workspace (set
// up by bella_op2d_set).
//
// The strips of all members (bella_strip2d.cuh), one after the other, are cut into equal runs,
// one for each warp of a cooperative launch of a block an SM, so a warp works on one member
// or on a few consecutive ones.  A phase of an iteration
//   P1  p = r + beta (p - omega v) on the fly, v = A p, <r^, v>
//   P2  s = r - alpha v on the fly,  t = A s,  <t,s>, <t,t>, <s,s>
//   P3  x += alpha p + omega s,  r = s - omega t,  <r^, r>, ||r||^2
// ends with each warp publishing its sums for each of its members in words that carry
// the number of the sum (SumWord, bella_iter2d.cuh).  A block goes on with a member when all of
// that member's words have come; that is all the waiting there is, since members have nothing
// to do with each other: no barrier over the grid, and the blocks of a member that has
// stopped are done.  Every block adds a member's words in the same order, so all of them
// derive the same scalars and the same stop.  The right-hand sides' norms, the scaling of the
// double-float systems to unit right-hand sides and back, and the FP64 residuals of all
// members (k_batch_resid) are taken in one launch too, in place of six launches a member.
//
// 48 members of 161x81, 321x161 and 641x321 nodes, 8 iterations in double-float with the true
// residuals: 7.0 -> 2.1 ms; an iteration 470 -> 178 us (its traffic alone takes 121), in FP64
// 357; the residuals 860 -> 128 us.
#include <chrono>
#include <cstring>
#include <type_traits>
#include <mutex>
#include <string>
#include <vector>

#include "bella_internal.cuh"
#include "bella_iter2d.cuh"

namespace bella {

template <typename T> struct Num;
template <> struct Num<double> {
    static __device__ __forceinline__ double from(double d) { return d; }
    static __device__ __forceinline__ double to(double v) { return v; }
};
template <> struct Num<dfloat> {
    static __device__ __forceinline__ dfloat from(double d) { return dfloat(d); }
    static __device__ __forceinline__ double to(dfloat v) { return v.to_double(); }
};

template <typename T>
struct BMember {
    Op2D<T> op;
    int cross, has_hc;
    int vec;                   // every vector 16-byte aligned
    int add;                   // the solution is added to xout (a refinement)
    const double *b;
    T *x, *r, *rh, *p[2], *v[2], *t;
    double *xout;              // FP64 solution (== x for FP64 members)
    double rtol;               // relative tolerance of this member (||r|| <= rtol ||b||, or atol)
    int strip0, nstrips;       // its strips among all members'
    int seg0, nseg;            // its words: one for each warp that has strips of it
};

struct BState {
    double bnorm;
    int iter, done, status, detail;
};

// a block's own copy of the state of a member that it works on
struct BLoc {
    double rho, rho0, alpha, beta, omega, atol, bnorm;
    int active, early, iter;
    int zero;                  // the solution is zero
};

template <typename T>
struct BArgs {
    const BMember<T> *mem;
    BState *st;
    BLoc *loc;                 // for blocks with more members than BATCH_LOCS: block b's from first member + b
    SumWord *words;            // two sets (by the sum's parity) of three quantities
    int *err;                  // 1: a wait gave up
    int nmem, strips, segs, h;
    double tol, atol_user;
    int maxiter;
    int legacy;                // scipy 1.7 legacy exit ||b|| <= tol (off for refinement solves)
};

constexpr int BATCH_WARPS = 16, BATCH_LOCS = 32;

// n things in k consecutive runs: where run i begins, and the run that thing s is in
__host__ __device__ inline int run_begin(int n, int i, int k) { return (int)((long long)n * i / k); }
__host__ __device__ inline int run_of(int n, int s, int k) { return (int)(((long long)(s + 1) * k - 1) / n); }

// The number, among the warps that have strips, of the one that has strip s of n, for `blocks`
// (at most n) blocks of `warps`: runs for blocks, and in those for warps, none empty.
__host__ __device__ inline int warp_of_strip(int n, int s, int blocks, int warps) {
    if ((long long)n < (long long)blocks * warps) return s;     // a strip a warp
    const int b = run_of(n, s, blocks), s0 = run_begin(n, b, blocks);
    return b * warps + run_of(run_begin(n, b + 1, blocks) - s0, s - s0, warps);
}

template <typename T>
__device__ int member_of(const BMember<T> *mem, int nmem, int strip) {
    int lo = 0, hi = nmem - 1;     // members are in strip order
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (mem[mid].strip0 <= strip) lo = mid; else hi = mid - 1;
    }
    return lo;
}

// this warp's strips s0 .. s1-1, its first member and the word that it has for member m, seg + m
struct WarpRun {
    int s0, s1, m, seg;
};
template <typename T>
__device__ WarpRun warp_run(const BMember<T> *mem, int nmem, int strips, int warps) {
    const int b = blockIdx.x, G = gridDim.x, w = threadIdx.x >> 5;
    const int b0 = run_begin(strips, b, G), nb = run_begin(strips, b + 1, G) - b0, nw = nb < warps ? nb : warps;
    WarpRun r = {0, 0, 0, 0};
    if (w < nw) {
        r.s0 = b0 + run_begin(nb, w, nw);
        r.s1 = b0 + run_begin(nb, w + 1, nw);
        r.m = member_of(mem, nmem, r.s0);
        r.seg = warp_of_strip(strips, r.s0, G, warps);
    }
    return r;
}
// f(member, its number, strips a .. e-1 of it) for every member of the warp's run
template <typename T, class F>
__device__ __forceinline__ void each_member(const WarpRun &r, const BMember<T> *mem, F f) {
    int m = r.m;
    for (int s = r.s0; s < r.s1; ++m) {
        const BMember<T> &M = mem[m];
        const int end = M.strip0 + M.nstrips, e = end < r.s1 ? end : r.s1;
        f(M, m, s - M.strip0, e - M.strip0);
        s = e;
    }
}
// the share of a member's nodes that goes with its strips a .. e-1: lo even
template <typename T>
__device__ __forceinline__ void node_range(const BMember<T> &M, int a, int e, long long &lo, long long &hi) {
    const long long n = (long long)M.op.nx * M.op.ny;
    lo = 2 * ((n / 2) * a / M.nstrips);
    hi = e == M.nstrips ? n : 2 * ((n / 2) * e / M.nstrips);
}

// a warp's sums of one member
template <int Q>
__device__ __forceinline__ void publish(SumWord *words, int segs, int seg, double (&v)[Q], unsigned long long seq) {
#pragma unroll
    for (int q = 0; q < Q; ++q) v[q] = warp_sum(v[q]);
    __syncwarp();                      // the warp's writes come before lane 0's fence
    if ((threadIdx.x & 31) == 0) {
        __threadfence();
#pragma unroll
        for (int q = 0; q < Q; ++q) sum_publish(words + ((size_t)(seq & 1) * 3 + q) * segs + seg, v[q], seq);
    }
}

// The Q totals of sum seq for each of this block's active members, given to fin(member's place
// in the block, totals) of one thread; false: a word did not come.  As many members at once as
// there are warps for.  A sum's words go in four parts, each added in a fixed order, so that
// every block gets the same total; as many warps read them as there are for it, since a word
// waits behind the others of its lane.
constexpr int SUM_PARTS = 4;
template <typename T, int Q, class Fin>
__device__ __forceinline__ bool totals(const BArgs<T> &A, const BLoc *loc, int m0, int nloc, unsigned long long seq,
                                       double *red, Fin fin) {
    const int w = threadIdx.x >> 5, lane = threadIdx.x & 31;
    for (int l0 = 0; l0 < nloc; l0 += BATCH_WARPS / Q) {
        const int nl = nloc - l0 < BATCH_WARPS / Q ? nloc - l0 : BATCH_WARPS / Q;
        const int room = BATCH_WARPS / (nl * Q), tw = room >= 4 ? 4 : room >= 2 ? 2 : 1, pair = w / tw;   // warps a sum
        bool ok = true;
        if (pair < nl * Q && loc[l0 + pair / Q].active) {
            const BMember<T> &M = A.mem[m0 + l0 + pair / Q];
            const int nseg = M.nseg;
            const SumWord *set = A.words + ((size_t)(seq & 1) * 3 + pair % Q) * A.segs + M.seg0;
            for (int part = w - pair * tw; part < SUM_PARTS; part += tw) {
                double s = 0.0;
                if (part * 32 < nseg) {
                    for (int i = part * 32 + lane; i < nseg && ok; i += SUM_PARTS * 32) {
                        double x;
                        unsigned long long got;
                        int spins = 0;
                        for (;;) {
                            sum_read(set + i, x, got);
                            if (got == seq) break;
                            if (++spins > SUM_SPIN_LIMIT) {
                                ok = false;
                                break;
                            }
                        }
                        s += x;
                    }
                    __syncwarp();
                    s = warp_sum(s);
                }
                if (lane == 0) red[pair * SUM_PARTS + part] = s;
            }
        }
        if (!__syncthreads_and(ok)) {
            if (threadIdx.x == 0) atomicExch(A.err, 1);
            return false;
        }
        if (w < nl && lane == 0 && loc[l0 + w].active) {
            double tot[Q];
#pragma unroll
            for (int q = 0; q < Q; ++q) {
                const double *p = red + (w * Q + q) * SUM_PARTS;
                tot[q] = (p[0] + p[1]) + (p[2] + p[3]);
            }
            fin(l0 + w, tot);
        }
        __syncthreads();
    }
    return true;
}

// P1 (M_PDIR) and P2 (M_SDIR) on strips a .. e-1 of a member
template <typename T, int MODE, bool CROSS, bool HC>
__device__ __forceinline__ void member_strips(const BMember<T> &M, const BLoc &L, int h, int a, int e,
                                              typename LaneAcc<T>::type (&acc)[3]) {
    StArgs<T> s = {};
    s.r = M.r; s.rh = M.rh; s.y = M.t;
    s.p0 = M.p[0]; s.p1 = M.p[1]; s.v0 = M.v[0]; s.v1 = M.v[1];
    stencil_phase<T, MODE, CROSS, HC, true>(M.op, s, h, L.iter, Num<T>::from(L.alpha), Num<T>::from(L.beta),
                                            Num<T>::from(L.omega), a, e, 1, acc[0], acc[1], acc[2]);
}

// CROSS: some member has Coriolis cross terms
template <typename T, bool CROSS>
__global__ void __launch_bounds__(BATCH_WARPS * 32, 1)
k_batch_bicgstab(BArgs<T> A) {
    __shared__ BLoc sloc[BATCH_LOCS];
    __shared__ double red[BATCH_WARPS * SUM_PARTS];
    const int lane = threadIdx.x & 31;
    const int b0 = run_begin(A.strips, blockIdx.x, gridDim.x), b1 = run_begin(A.strips, blockIdx.x + 1, gridDim.x);
    const int m0 = member_of(A.mem, A.nmem, b0), nloc = member_of(A.mem, A.nmem, b1 - 1) - m0 + 1;
    BLoc *loc = nloc <= BATCH_LOCS ? sloc : A.loc + m0 + blockIdx.x;
    const WarpRun run = warp_run(A.mem, A.nmem, A.strips, BATCH_WARPS);
    for (int l = threadIdx.x; l < nloc; l += blockDim.x) {
        BLoc L = {};
        L.active = 1;
        loc[l] = L;
    }
    __syncthreads();
    // member l of the block stops; the block with its first strip records it
    auto stop = [&](int l, int status, int detail) {
        BLoc &L = loc[l];
        L.active = 0;
        if (A.mem[m0 + l].strip0 >= b0) {
            BState S;
            S.bnorm = L.bnorm;
            S.iter = L.iter;
            S.done = 1;
            S.status = status;
            S.detail = detail;
            A.st[m0 + l] = S;
        }
    };
    unsigned long long seq = 0;
    if (!std::is_same<T, double>::value) {
        // Double-float has the FP32 exponent range: a member solves its system scaled to a unit
        // right-hand side (BiCGStab is scale-invariant).  ||b|| in FP64
        ++seq;
        each_member(run, A.mem, [&](const BMember<T> &M, int m, int a, int e) {
            long long lo, hi;
            node_range(M, a, e, lo, hi);
            DD s;
            s.zero();
#pragma unroll 4
            for (long long i = lo + lane; i < hi; i += 32) s.add_prod(M.b[i], M.b[i]);
            double v[1] = {s.value()};
            publish<1>(A.words, A.segs, run.seg + m, v, seq);
        });
        if (!totals<T, 1>(A, loc, m0, nloc, seq, red, [&](int l, const double (&tot)[1]) {
                BLoc &L = loc[l];
                L.bnorm = sqrt(tot[0]);
                if (!isfinite(L.bnorm)) {                                         // x0, as in FP64
                    L.zero = 1;
                    stop(l, BELLA_NONFINITE, 0);
                } else if (L.bnorm == 0.0 || (A.legacy && L.bnorm <= A.tol)) {    // scipy 1.7 legacy exit
                    L.zero = 1;
                    stop(l, BELLA_OK, 0);
                }
            }))
            return;
    }
    // r = r^ = b, x = 0, <b, b>
    ++seq;
    each_member(run, A.mem, [&](const BMember<T> &M, int m, int a, int e) {
        const BLoc &L = loc[m - m0];
        if (!L.active) return;
        const double scale = std::is_same<T, double>::value ? 1.0 : 1.0 / L.bnorm;
        long long lo, hi;
        node_range(M, a, e, lo, hi);
        typename Acc<T>::type s;
        s.zero();
#pragma unroll 4
        for (long long i = lo + lane; i < hi; i += 32) {
            const T bg = Num<T>::from(std::is_same<T, double>::value ? M.b[i] : scale * M.b[i]);
            M.r[i] = bg;
            M.rh[i] = bg;
            M.x[i] = Num<T>::from(0.0);
            s.add_prod(bg, bg);
        }
        double v[1] = {s.value()};
        publish<1>(A.words, A.segs, run.seg + m, v, seq);
    });
    if (!totals<T, 1>(A, loc, m0, nloc, seq, red, [&](int l, const double (&tot)[1]) {
            BLoc &L = loc[l];
            const double norm = sqrt(tot[0]);
            double rtol = A.mem[m0 + l].rtol;
            if (std::is_same<T, double>::value) {
                L.bnorm = norm;
                L.atol = rtol * norm;
                if (A.atol_user > L.atol) L.atol = A.atol_user;
            } else {
                if (A.atol_user / L.bnorm > rtol) rtol = A.atol_user / L.bnorm;
                L.atol = rtol * norm;
            }
            L.rho = L.rho0 = tot[0];
            L.alpha = L.omega = 1.0;
            if (!isfinite(tot[0])) stop(l, BELLA_NONFINITE, 0);
            else if (norm == 0.0 || (std::is_same<T, double>::value && A.legacy && norm <= A.tol)) stop(l, BELLA_OK, 0);
            else if (A.maxiter <= 0) stop(l, BELLA_MAXITER, 0);
        }))
        return;
    const double eps2 = 4.930380657631324e-32;
    for (;;) {
        int any = 0;
        for (int l = threadIdx.x; l < nloc; l += blockDim.x) any |= loc[l].active;
        if (!__syncthreads_or(any)) break;
        // ---- P1: p and v = A p, <r^, v>; alpha
        ++seq;
        each_member(run, A.mem, [&](const BMember<T> &M, int m, int a, int e) {
            const BLoc &L = loc[m - m0];
            if (!L.active) return;
            typename LaneAcc<T>::type acc[3];
            acc[0].zero(); acc[1].zero(); acc[2].zero();
            if (CROSS && M.cross) {
                if (M.has_hc) member_strips<T, M_PDIR, CROSS, true>(M, L, A.h, a, e, acc);
                else member_strips<T, M_PDIR, CROSS, false>(M, L, A.h, a, e, acc);
            } else {
                if (M.has_hc) member_strips<T, M_PDIR, false, true>(M, L, A.h, a, e, acc);
                else member_strips<T, M_PDIR, false, false>(M, L, A.h, a, e, acc);
            }
            double v[1] = {acc[0].value()};
            publish<1>(A.words, A.segs, run.seg + m, v, seq);
        });
        if (!totals<T, 1>(A, loc, m0, nloc, seq, red, [&](int l, const double (&tot)[1]) {
                if (!isfinite(tot[0])) stop(l, BELLA_NONFINITE, 0);
                else if (tot[0] == 0.0) stop(l, BELLA_BREAKDOWN, 3);
                else loc[l].alpha = loc[l].rho / tot[0];
            }))
            return;
        // ---- P2: s and t = A s, <t,s>, <t,t>, <s,s>; omega (early exit on ||s||)
        ++seq;
        each_member(run, A.mem, [&](const BMember<T> &M, int m, int a, int e) {
            const BLoc &L = loc[m - m0];
            if (!L.active) return;
            typename LaneAcc<T>::type acc[3];
            acc[0].zero(); acc[1].zero(); acc[2].zero();
            if (CROSS && M.cross) {
                if (M.has_hc) member_strips<T, M_SDIR, CROSS, true>(M, L, A.h, a, e, acc);
                else member_strips<T, M_SDIR, CROSS, false>(M, L, A.h, a, e, acc);
            } else {
                if (M.has_hc) member_strips<T, M_SDIR, false, true>(M, L, A.h, a, e, acc);
                else member_strips<T, M_SDIR, false, false>(M, L, A.h, a, e, acc);
            }
            double v[3] = {acc[0].value(), acc[1].value(), acc[2].value()};
            publish<3>(A.words, A.segs, run.seg + m, v, seq);
        });
        if (!totals<T, 3>(A, loc, m0, nloc, seq, red, [&](int l, const double (&tot)[3]) {
                BLoc &L = loc[l];
                const double ts = tot[0], tt = tot[1], ss = tot[2];
                if (!isfinite(ss) || !isfinite(ts) || !isfinite(tt)) stop(l, BELLA_NONFINITE, 0);
                else if (sqrt(ss) <= L.atol) L.early = 1;
                else if (!(tt > 0.0)) stop(l, BELLA_BREAKDOWN, 4);
                else L.omega = ts / tt;
            }))
            return;
        // ---- P3: x and r, <r^, r>, ||r||^2; the stop tests and beta
        ++seq;
        each_member(run, A.mem, [&](const BMember<T> &M, int m, int a, int e) {
            const BLoc &L = loc[m - m0];
            if (!L.active) return;
            long long lo, hi;
            node_range(M, a, e, lo, hi);
            const bool odd = L.iter & 1;               // p and v written by this iteration's P1
            T *x = M.x + lo, *r = M.r + lo;
            const T *p = (odd ? M.p[0] : M.p[1]) + lo, *v = (odd ? M.v[0] : M.v[1]) + lo;
            const T alpha = Num<T>::from(L.alpha), omega = Num<T>::from(L.omega);
            typename Acc<T>::type u0, u1;
            u0.zero(); u1.zero();
            if (M.vec)
                update_phase<T, true, true>(hi - lo, x, p, r, v, M.t + lo, M.rh + lo, alpha, omega, L.early != 0, lane,
                                            32, u0, u1);
            else
                update_phase<T, false, true>(hi - lo, x, p, r, v, M.t + lo, M.rh + lo, alpha, omega, L.early != 0, lane,
                                             32, u0, u1);
            double s[2] = {u0.value(), u1.value()};
            publish<2>(A.words, A.segs, run.seg + m, s, seq);
        });
        if (!totals<T, 2>(A, loc, m0, nloc, seq, red, [&](int l, const double (&tot)[2]) {
                BLoc &L = loc[l];
                ++L.iter;
                if (L.early) stop(l, BELLA_OK, 0);
                else if (!isfinite(tot[0]) || !isfinite(tot[1])) stop(l, BELLA_NONFINITE, 0);
                else if (sqrt(tot[1]) <= L.atol) stop(l, BELLA_OK, 0);
                else if (L.iter >= A.maxiter) stop(l, BELLA_MAXITER, 0);
                else if (fabs(tot[0]) < eps2 * L.rho0) stop(l, BELLA_BREAKDOWN, 1);
                else if (fabs(L.omega) < eps2) stop(l, BELLA_BREAKDOWN, 2);
                else {
                    L.beta = (tot[0] / L.rho) * (L.alpha / L.omega);
                    L.rho = tot[0];
                }
            }))
            return;
    }
    // the FP64 solution of double-float members, scaled back (each warp the nodes that it updated)
    if (!std::is_same<T, double>::value) {
        each_member(run, A.mem, [&](const BMember<T> &M, int m, int a, int e) {
            const BLoc &L = loc[m - m0];
            long long lo, hi;
            node_range(M, a, e, lo, hi);
#pragma unroll 4
            for (long long i = lo + lane; i < hi; i += 32) {
                const double x = L.zero ? 0.0 : L.bnorm * Num<T>::to(ld_vec<true>(M.x + i));
                M.xout[i] = M.add ? M.xout[i] + x : x;
            }
        });
    }
}

// r = b - A x in FP64 for every member (r: M.r, x: M.x), and ||r||^2 by warps and members in sums
template <bool CROSS>
__global__ void __launch_bounds__(NTHREADS, 4)
k_batch_resid(const BMember<double> *mem, int nmem, int strips, int h, double *sums) {
    const WarpRun run = warp_run(mem, nmem, strips, NTHREADS / 32);
    each_member(run, mem, [&](const BMember<double> &M, int m, int a, int e) {
        StArgs<double> s = {};
        s.x = M.x; s.b = M.b; s.y = M.r;
        LaneAcc<double>::type c0, c1, c2;
        c0.zero(); c1.zero(); c2.zero();
        if (CROSS && M.cross) {
            if (M.has_hc) stencil_phase<double, M_RESID, CROSS, true, false>(M.op, s, h, 0, 0., 0., 0., a, e, 1, c0, c1, c2);
            else stencil_phase<double, M_RESID, CROSS, false, false>(M.op, s, h, 0, 0., 0., 0., a, e, 1, c0, c1, c2);
        } else {
            if (M.has_hc) stencil_phase<double, M_RESID, false, true, false>(M.op, s, h, 0, 0., 0., 0., a, e, 1, c0, c1, c2);
            else stencil_phase<double, M_RESID, false, false, false>(M.op, s, h, 0, 0., 0., 0., a, e, 1, c0, c1, c2);
        }
        const double v = warp_sum(c0.value());
        if ((threadIdx.x & 31) == 0) sums[run.seg + m] = v;
    });
}

// ---------------------------------------------------------------------------
// host side: launch configurations and the autotuner
// ---------------------------------------------------------------------------
// rows of a strip; 0: by the members' sizes (best_strip_height)
static const int kConfigs[] = {0, 4, 8, 12, 16, 32};
constexpr int NCONFIG = (int)(sizeof(kConfigs) / sizeof(kConfigs[0]));

// a device buffer that grows
struct DevBuf {
    void *p = nullptr;
    size_t cap = 0;
    bool reserve(size_t bytes) {
        if (bytes <= cap) return true;
        cudaFree(p);
        p = nullptr;
        cap = 0;
        if (cudaMalloc(&p, bytes) != cudaSuccess) return false;
        cap = bytes;
        return true;
    }
};

struct BatchCtx {
    DevBuf mem, st, loc, words, err;      // a launch's BMember<T>[], BState[], BLoc[], SumWord[] and error flag
    DevBuf rmem, rsum;                    // the residuals' members and sums
    DevBuf save;                          // a member's iterate kept while it is finished alone
    // autotuned choice per member-size signature
    std::vector<std::pair<std::string, int>> tuned;
};

static std::mutex g_batch_mu;
static BatchCtx g_batch[64];

static std::string signature(bella_ws *const *ws, int nmem) {
    std::string s;
    for (int m = 0; m < nmem; ++m) s += std::to_string(ws[m]->nx) + "x" + std::to_string(ws[m]->ny) + ";";
    return s;
}

template <typename T> static void member_vectors(BMember<T> &M, bella_ws *w, double *x);
template <> void member_vectors<double>(BMember<double> &M, bella_ws *w, double *x) {
    const size_t nc = (size_t)(w->nx + 1) * (w->ny + 1);
    M.op.axx = w->a64; M.op.ayy = w->a64 + nc; M.op.axy = w->a64 + 2 * nc; M.op.ayx = w->a64 + 3 * nc;
    M.op.dinv = w->dinv64; M.op.hc = w->hc64;
    M.x = x; M.xout = x; M.r = w->r64k; M.rh = w->rh64;
    M.p[0] = w->p64[0]; M.p[1] = w->p64[1]; M.v[0] = w->v64[0]; M.v[1] = w->v64[1]; M.t = w->t64;
}
template <> void member_vectors<dfloat>(BMember<dfloat> &M, bella_ws *w, double *x) {
    const size_t nc = (size_t)(w->nx + 1) * (w->ny + 1);
    M.op.axx = w->adf; M.op.ayy = w->adf + nc; M.op.axy = w->adf + 2 * nc; M.op.ayx = w->adf + 3 * nc;
    M.op.dinv = w->dinvdf; M.op.hc = w->hcdf;
    M.x = w->xdf; M.xout = x; M.r = w->rdf; M.rh = w->rhdf;
    M.p[0] = w->pdf[0]; M.p[1] = w->pdf[1]; M.v[0] = w->vdf[0]; M.v[1] = w->vdf[1]; M.t = w->tdf;
}

// the members' strips of h rows, cut up for `blocks` blocks of `warps` warps
template <typename T>
static int lay_out(std::vector<BMember<T>> &hm, int h, int sms, int per_sm, int warps, int &strips, int &segs) {
    long long total = 0;
    for (BMember<T> &M : hm) {
        const long long n = (long long)strips_across(M.op.nx, strip_width<T>()) * strips_down(M.op.ny, h);
        M.strip0 = (int)total;
        M.nstrips = (int)n;
        total += n;
    }
    if (total > 0x7fffffff) return 0;
    strips = (int)total;
    const int blocks = strips < sms * per_sm ? strips : sms * per_sm;
    segs = 0;
    for (size_t m = 0; m < hm.size(); ++m) {
        BMember<T> &M = hm[m];
        const int w0 = warp_of_strip(strips, M.strip0, blocks, warps);
        const int w1 = warp_of_strip(strips, M.strip0 + M.nstrips - 1, blocks, warps);
        M.seg0 = (int)m + w0;
        M.nseg = w1 - w0 + 1;
        segs = M.seg0 + M.nseg;
    }
    return blocks;
}

// rows of a strip; from the first 64 sizes where there are more
template <typename T>
static int rows_of(const std::vector<BMember<T>> &hm, int sms, int warps_per_sm) {
    struct Size { int across, ny, count; };
    std::vector<Size> sizes;               // an ensemble has many members of few sizes
    for (const BMember<T> &M : hm) {
        const int across = strips_across(M.op.nx, strip_width<T>());
        size_t q = 0;
        while (q < sizes.size() && (sizes[q].across != across || sizes[q].ny != M.op.ny)) ++q;
        if (q == sizes.size() && q < 64) sizes.push_back({across, M.op.ny, 0});
        if (q < sizes.size()) sizes[q].count++;
    }
    return best_strip_height<T>([&](int h) {
        long long n = 0;
        for (const Size &z : sizes) n += (long long)z.count * z.across * strips_down(z.ny, h);
        return n;
    }, sms, warps_per_sm);
}

// one launch with configuration cfg; fills per-member results.  rtol (each member's own tolerance): a
// refinement, whose solutions are added to x
template <typename T>
static int batch_run(BatchCtx &c, bella_ws *const *ws, int nmem, const double *const *b, double *const *x,
                     const bella_solve_opts &o, int cfg, cudaStream_t s, std::vector<BState> *out, const double *rtol) {
    std::vector<BMember<T>> hm(nmem);
    bool cross = false;
    for (int m = 0; m < nmem; ++m) {
        bella_ws *w = ws[m];
        BMember<T> &M = hm[m];
        M = {};
        M.op.nx = w->nx; M.op.ny = w->ny;
        member_vectors<T>(M, w, x[m]);
        M.b = b[m];
        M.cross = w->cross; M.has_hc = w->has_hc;
        M.vec = reinterpret_cast<uintptr_t>(M.x) % 16 == 0;      // x may be the caller's; the others are aligned
        M.add = rtol != nullptr;
        M.rtol = rtol ? rtol[m] : o.tol;
        cross = cross || w->cross;
    }
    void (*kern)(BArgs<T>) = cross ? k_batch_bicgstab<T, true> : k_batch_bicgstab<T, false>;
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, kern, BATCH_WARPS * 32, 0) != cudaSuccess || per_sm < 1)
        return BELLA_ECUDA;
    const int sms = num_sms();
    BArgs<T> A;
    A.h = kConfigs[cfg] ? kConfigs[cfg] : rows_of(hm, sms, BATCH_WARPS);
    const int grid = lay_out(hm, A.h, sms, 1, BATCH_WARPS, A.strips, A.segs);
    if (grid < 1) return BELLA_EINVAL;
    const size_t words = (size_t)6 * A.segs * sizeof(SumWord);
    if (!c.mem.reserve(nmem * sizeof(BMember<T>)) || !c.st.reserve(nmem * sizeof(BState)) ||
        !c.loc.reserve((size_t)(nmem + grid) * sizeof(BLoc)) || !c.words.reserve(words) || !c.err.reserve(sizeof(int)))
        return BELLA_ECUDA;
    if (cudaMemcpyAsync(c.mem.p, hm.data(), nmem * sizeof(BMember<T>), cudaMemcpyHostToDevice, s) != cudaSuccess ||
        cudaMemsetAsync(c.st.p, 0, nmem * sizeof(BState), s) != cudaSuccess ||
        cudaMemsetAsync(c.words.p, 0, words, s) != cudaSuccess ||
        cudaMemsetAsync(c.err.p, 0, sizeof(int), s) != cudaSuccess)
        return BELLA_ECUDA;
    A.mem = (const BMember<T> *)c.mem.p; A.st = (BState *)c.st.p; A.loc = (BLoc *)c.loc.p;
    A.words = (SumWord *)c.words.p; A.err = (int *)c.err.p;
    A.nmem = nmem;
    A.tol = o.tol; A.atol_user = rtol ? 0.0 : o.atol; A.maxiter = o.maxiter;
    A.legacy = rtol == nullptr;
    void *args[] = {&A};
    if (cudaLaunchCooperativeKernel((const void *)kern, grid, BATCH_WARPS * 32, args, 0, s) != cudaSuccess)
        return BELLA_ECUDA;
    if (out) {
        out->resize(nmem);
        int err = 0;
        if (cudaMemcpyAsync(out->data(), c.st.p, nmem * sizeof(BState), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaMemcpyAsync(&err, c.err.p, sizeof(int), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
            cudaStreamSynchronize(s) != cudaSuccess)
            return BELLA_ECUDA;
        if (err) return BELLA_ECUDA;   // a member's sums did not come (bounded wait)
    }
    return BELLA_OK;
}

static int batch_run_prec(int prec, BatchCtx &c, bella_ws *const *ws, int nmem, const double *const *b,
                          double *const *x, const bella_solve_opts &o, int cfg, cudaStream_t s,
                          std::vector<BState> *out, const double *rtol = nullptr) {
    if (prec == 0) return batch_run<double>(c, ws, nmem, b, x, o, cfg, s, out, rtol);
    return batch_run<dfloat>(c, ws, nmem, b, x, o, cfg, s, out, rtol);
}

// the FP64 residuals of all members in their r64, and ||r||^2 of each (synchronises)
static int batch_resid(BatchCtx &c, bella_ws *const *ws, int nmem, const double *const *b, double *const *x,
                       cudaStream_t s, std::vector<double> &rr) {
    std::vector<BMember<double>> hm(nmem);
    bool cross = false;
    for (int m = 0; m < nmem; ++m) {
        BMember<double> &M = hm[m];
        M = {};
        M.op.nx = ws[m]->nx; M.op.ny = ws[m]->ny;
        member_vectors<double>(M, ws[m], x[m]);
        M.r = ws[m]->r64;
        M.b = b[m];
        M.cross = ws[m]->cross; M.has_hc = ws[m]->has_hc;
        cross = cross || ws[m]->cross;
    }
    constexpr int per_sm = 4, warps = NTHREADS / 32;
    const int sms = num_sms(), h = rows_of(hm, sms, per_sm * warps);
    int strips = 0, segs = 0;
    const int grid = lay_out(hm, h, sms, per_sm, warps, strips, segs);
    if (grid < 1) return BELLA_EINVAL;
    if (!c.rmem.reserve(nmem * sizeof(BMember<double>)) || !c.rsum.reserve(segs * sizeof(double))) return BELLA_ECUDA;
    if (cudaMemcpyAsync(c.rmem.p, hm.data(), nmem * sizeof(BMember<double>), cudaMemcpyHostToDevice, s) != cudaSuccess)
        return BELLA_ECUDA;
    const BMember<double> *mem = (const BMember<double> *)c.rmem.p;
    if (cross) k_batch_resid<true><<<grid, NTHREADS, 0, s>>>(mem, nmem, strips, h, (double *)c.rsum.p);
    else k_batch_resid<false><<<grid, NTHREADS, 0, s>>>(mem, nmem, strips, h, (double *)c.rsum.p);
    std::vector<double> sums(segs);
    if (cudaGetLastError() != cudaSuccess ||
        cudaMemcpyAsync(sums.data(), c.rsum.p, segs * sizeof(double), cudaMemcpyDeviceToHost, s) != cudaSuccess ||
        cudaStreamSynchronize(s) != cudaSuccess)
        return BELLA_ECUDA;
    rr.assign(nmem, 0.0);
    for (int m = 0; m < nmem; ++m)
        for (int q = 0; q < hm[m].nseg; ++q) rr[m] += sums[hm[m].seg0 + q];
    return BELLA_OK;
}

static int check_members(bella_ws *const *ws, int nmem, const double *const *b, double *const *x) {
    if (!ws || !b || !x || nmem < 1) return BELLA_EINVAL;
    for (int m = 0; m < nmem; ++m) {
        if (!ws[m] || !b[m] || !x[m]) return BELLA_EINVAL;
        if (ws[m]->ndim != 2) return BELLA_ENOOP;
        if (ws[m]->ymirror) return BELLA_EINVAL;     // the batched stencil wraps y (no LAMB_BDRY mirror)
        if (ws[m]->device != ws[0]->device) return BELLA_EINVAL;
    }
    return BELLA_OK;
}

}  // namespace bella

using namespace bella;

extern "C" {

// Autotuner: times every launch configuration on maxiter_probe iterations of
// the batch and keeps the fastest for this set of member sizes.  *choice
// (optional) receives its index; *ms (optional, NCONFIG entries) the times.
int bella_batch_autotune(bella_ws *const *ws, int nmembers, const double *const *b, double *const *x,
                         int precision, int probe_iters, int *choice, double *ms, void *stream) {
    const int prec = precision == 0 ? 0 : 2;
    int rc = check_members(ws, nmembers, b, x);
    if (rc != BELLA_OK) return rc;
    std::lock_guard<std::mutex> lk(g_batch_mu);
    const int dev = ws[0]->device;
    if (dev < 0 || dev >= 64) return BELLA_EINVAL;
    if (cudaSetDevice(dev) != cudaSuccess) return BELLA_ECUDA;
    BatchCtx &c = g_batch[dev];
    cudaStream_t s = (cudaStream_t)stream;
    bella_solve_opts o;
    bella_solve_opts_default(&o);
    o.tol = 0.0;
    o.maxiter = probe_iters > 0 ? probe_iters : 20;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    int best = 0;
    float best_ms = 1e30f;
    for (int cfg = 0; cfg < NCONFIG; ++cfg) {
        float t = 0.f;
        for (int rep = 0; rep < 2; ++rep) {   // first run warms up
            cudaEventRecord(e0, s);
            rc = batch_run_prec(prec, c, ws, nmembers, b, x, o, cfg, s, nullptr);
            if (rc != BELLA_OK) break;
            cudaEventRecord(e1, s);
            if (cudaEventSynchronize(e1) != cudaSuccess) { rc = BELLA_ECUDA; break; }
            cudaEventElapsedTime(&t, e0, e1);
        }
        if (rc != BELLA_OK) break;
        if (ms) ms[cfg] = t;
        if (t < best_ms) { best_ms = t; best = cfg; }
    }
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    if (rc != BELLA_OK) return rc;
    const std::string sig = signature(ws, nmembers) + (prec == 0 ? "fp64" : "df64");
    bool found = false;
    for (auto &p : c.tuned)
        if (p.first == sig) { p.second = best; found = true; }
    if (!found) c.tuned.emplace_back(sig, best);
    if (choice) *choice = best;
    return BELLA_OK;
}

int bella_batch_config_count(void) { return NCONFIG; }

int bella_batch_config(int index, int *tile_x, int *tile_y, int *ctas_per_sm) {
    if (index < 0 || index >= NCONFIG) return BELLA_EINVAL;
    if (tile_x) *tile_x = strip_width<dfloat>();
    if (tile_y) *tile_y = kConfigs[index];
    if (ctas_per_sm) *ctas_per_sm = 1;
    return BELLA_OK;
}

// FP64 BiCGStab (scipy control flow, x0 = 0) for nmembers 2D systems in one
// persistent launch.  ws[m]: workspace with member m's operator
// (bella_op2d_set); b[m], x[m]: device FP64 vectors of its nx*ny nodes.
// opts: tol, atol, maxiter (shared); config < 0 takes the autotuned choice for
// these member sizes (the first configuration when none was tuned).
// stats[m] (optional): iterations, status, detail, bnorm and the true FP64
// relative residual.  Returns BELLA_OK when every member converged, else the
// first non-OK member status; BELLA_ECUDA if a wait for a member's sums gave up.
int bella_bicgstab_batched(bella_ws *const *ws, int nmembers, const double *const *b, double *const *x,
                           const bella_solve_opts *opts, int config, bella_solve_stats *stats, void *stream) {
    int rc = check_members(ws, nmembers, b, x);
    if (rc != BELLA_OK) return rc;
    if (config >= NCONFIG) return BELLA_EINVAL;
    std::lock_guard<std::mutex> lk(g_batch_mu);
    const int dev = ws[0]->device;
    if (dev < 0 || dev >= 64) return BELLA_EINVAL;
    if (cudaSetDevice(dev) != cudaSuccess) return BELLA_ECUDA;
    BatchCtx &c = g_batch[dev];
    cudaStream_t s = (cudaStream_t)stream;
    const auto t0 = std::chrono::steady_clock::now();
    bella_solve_opts o;
    if (opts) o = *opts; else bella_solve_opts_default(&o);
    if (!(o.tol >= 0.0) || o.maxiter < 0) return BELLA_EINVAL;
    const int prec = o.precision == 0 ? 0 : 2;
    int cfg = config;
    if (cfg < 0) {
        cfg = 0;
        const std::string sig = signature(ws, nmembers) + (prec == 0 ? "fp64" : "df64");
        for (auto &p : c.tuned)
            if (p.first == sig) cfg = p.second;
    }
    std::vector<int> status(nmembers, BELLA_OK), its(nmembers, 0), detail(nmembers, 0), rounds(nmembers, 0);
    std::vector<double> bnorm(nmembers, 0.0);
    std::vector<double> rr(nmembers);      // ||b - A x||^2 in FP64
    {
        std::vector<BState> res;
        rc = batch_run_prec(prec, c, ws, nmembers, b, x, o, cfg, s, &res);
        if (rc != BELLA_OK) return rc;
        for (int m = 0; m < nmembers; ++m) {
            status[m] = res[m].done ? res[m].status : BELLA_MAXITER;
            its[m] = res[m].iter;
            detail[m] = res[m].detail;
            bnorm[m] = res[m].bnorm;
        }
    }
    // FP64 true residuals; double-float members that converged on the recursion
    // but miss the tolerance in FP64 are refined: A d = r (x0 = 0) in a batched
    // launch of just those members, x += d, up to 4 rounds
    for (int round = 0;; ++round) {
        rc = batch_resid(c, ws, nmembers, b, x, s, rr);
        if (rc != BELLA_OK) return rc;
        if (prec == 0 || round >= 4) break;
        std::vector<bella_ws *> sw;
        std::vector<const double *> sb;
        std::vector<double *> sx;
        std::vector<double> rt;
        std::vector<int> idx;
        for (int m = 0; m < nmembers; ++m) {
            double target = o.tol * bnorm[m];
            if (o.atol > target) target = o.atol;
            const double r = sqrt(rr[m]);
            if (status[m] == BELLA_OK && isfinite(r) && r > target && r > 0.0) {
                idx.push_back(m);
                sw.push_back(ws[m]);
                sb.push_back(ws[m]->r64);
                sx.push_back(x[m]);
                rt.push_back(0.5 * target / r);
            }
        }
        if (idx.empty()) break;
        std::vector<BState> sub;
        rc = batch_run_prec(prec, c, sw.data(), (int)idx.size(), sb.data(), sx.data(), o, cfg, s, &sub, rt.data());
        if (rc != BELLA_OK) return rc;
        for (size_t q = 0; q < idx.size(); ++q) {
            const int m = idx[q];
            its[m] += sub[q].iter;
            rounds[m] += 1;
            if (!sub[q].done || sub[q].status != BELLA_OK) status[m] = sub[q].done ? sub[q].status : BELLA_MAXITER;
        }
    }
    // double-float members whose batched iteration broke down, or whose FP64 true
    // residual still misses the tolerance after the refinement rounds (the
    // double-float floor of a hard system), are finished one by one by the FP64
    // solve from their iterate, within the iteration budget left; the batched
    // iterate is kept unless that lowers its FP64 true residual.  Reported in
    // stats->fallback.
    std::vector<int> single(nmembers, 0);
    if (prec != 0) {
        bool any = false;
        for (int m = 0; m < nmembers; ++m) {
            double target = o.tol * bnorm[m];
            if (o.atol > target) target = o.atol;
            const double rm = sqrt(rr[m]);
            const bool missed = status[m] == BELLA_OK && isfinite(rm) && rm > target && !(bnorm[m] <= o.tol);
            if (!(status[m] == BELLA_BREAKDOWN || missed) || !isfinite(bnorm[m]) || !isfinite(rm) ||
                its[m] >= o.maxiter)
                continue;
            const long long nm_ = ws[m]->n;
            if (!c.save.reserve(nm_ * sizeof(double))) return BELLA_ECUDA;
            if (cudaMemcpyAsync(c.save.p, x[m], nm_ * sizeof(double), cudaMemcpyDeviceToDevice, s) != cudaSuccess)
                return BELLA_ECUDA;
            bella_solve_opts os = o;
            os.precision = 0;
            os.x0_zero = 0;
            os.maxiter = o.maxiter - its[m];
            bella_solve_stats fs;
            const int r = bella_bicgstab(ws[m], b[m], x[m], &os, &fs, stream);
            if (r < 0) return r;
            its[m] += fs.iterations;
            if (isfinite(fs.relres) && fs.relres * bnorm[m] < rm) {
                status[m] = fs.status;
                single[m] = 1;
            } else if (cudaMemcpyAsync(x[m], c.save.p, nm_ * sizeof(double), cudaMemcpyDeviceToDevice, s) !=
                       cudaSuccess) {
                return BELLA_ECUDA;
            }
            any = true;
        }
        if (any) {
            std::vector<KState> ks(nmembers);
            for (int m = 0; m < nmembers; ++m)
                if (single[m]) op2d_resid(ws[m], 0, x[m], b[m], ws[m]->r64, s);
            for (int m = 0; m < nmembers; ++m)
                if (single[m] && cudaMemcpyAsync(&ks[m], ws[m]->ks, sizeof(KState), cudaMemcpyDeviceToHost, s) != cudaSuccess)
                    return BELLA_ECUDA;
            if (cudaStreamSynchronize(s) != cudaSuccess) return BELLA_ECUDA;
            for (int m = 0; m < nmembers; ++m)
                if (single[m]) rr[m] = ks[m].dot_aux2;
        }
    }
    const double secs = std::chrono::duration<double>(std::chrono::steady_clock::now() - t0).count();
    int worst = BELLA_OK;
    for (int m = 0; m < nmembers; ++m) {
        double target = o.tol * bnorm[m];
        if (o.atol > target) target = o.atol;
        const double rn = sqrt(rr[m]);
        int st_m = status[m];
        if (st_m == BELLA_OK && !(rn <= target) && !(bnorm[m] <= o.tol)) st_m = BELLA_MAXITER;   // never on the recursion alone
        if (!isfinite(rn)) st_m = BELLA_NONFINITE;
        if (worst == BELLA_OK && st_m != BELLA_OK) worst = st_m;
        if (stats) {
            bella_solve_stats &q = stats[m];
            memset(&q, 0, sizeof(q));
            q.status = st_m;
            q.iterations = its[m];
            q.matvecs = 2 * its[m];
            q.bnorm = bnorm[m];
            q.relres = bnorm[m] > 0 ? rn / bnorm[m] : rn;
            q.seconds = secs;
            q.detail = detail[m];
            q.outer = cfg;
            q.fallback = rounds[m] + (single[m] ? 256 : 0);   // FP64 refinement rounds; +256: finished alone
        }
    }
    return worst;
}

}  // extern "C"
