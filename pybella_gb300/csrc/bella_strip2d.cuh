// bella_strip2d.cuh -- the 2D 9-point operator on a strip of nodes, one warp.
//
// A warp owns 30 node columns (double-float: 62, two to a lane), its outer columns carry the
// neighbours, and it marches down `h` rows: a lane keeps its column's last u, the cell to
// its right gets its flux from two rows of u (the right neighbour's by shuffle), and a node
// sums its four cells (the left ones' by shuffle).  Nothing goes through shared memory and
// nothing waits for another warp.  The arithmetic of a node is that of the cell-flux form
// in bella_op2d.cu, operation by operation.
#pragma once
#include "bella_internal.cuh"

namespace bella {

__device__ __forceinline__ float shfl_down1(float v) { return __shfl_down_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double shfl_down1(double v) { return __shfl_down_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ dfloat shfl_down1(dfloat v) { return dfloat(shfl_down1(v.hi), shfl_down1(v.lo)); }
__device__ __forceinline__ float shfl_up1(float v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ double shfl_up1(double v) { return __shfl_up_sync(0xffffffffu, v, 1); }
__device__ __forceinline__ dfloat shfl_up1(dfloat v) { return dfloat(shfl_up1(v.hi), shfl_up1(v.lo)); }

// loads of vectors: CG (from L2) where another block of the same launch writes them
template <bool CG> __device__ __forceinline__ float ld_vec(const float *p) { return CG ? __ldcg(p) : *p; }
template <bool CG> __device__ __forceinline__ double ld_vec(const double *p) { return CG ? __ldcg(p) : *p; }
template <bool CG> __device__ __forceinline__ dfloat ld_vec(const dfloat *p) {
    if (!CG) return *p;
    const float2 v = __ldcg(reinterpret_cast<const float2 *>(p));
    return dfloat(v.x, v.y);
}

// The values of one or two neighbouring columns that a lane works on: FP64 and FP32 one at a
// time, double-float two (packed FP32 instructions).  A strip has 32 V columns, the outer
// two its neighbours.
template <typename T> struct Lane {                    // V = 1
    typedef T V;
    static constexpr int N = 1;
    static __device__ __forceinline__ V splat(T a) { return a; }
    static __device__ __forceinline__ V join(const T (&a)[1]) { return a[0]; }
    static __device__ __forceinline__ void split(V v, T (&a)[1]) { a[0] = v; }
    static __device__ __forceinline__ V right(V v) { return shfl_down1(v); }      // each column's right neighbour
    static __device__ __forceinline__ V left(V v) { return shfl_up1(v); }
};
template <> struct Lane<dfloat> {
    typedef dfloat2 V;
    static constexpr int N = 2;
    static __device__ __forceinline__ V splat(dfloat a) { return dfloat2(a, a); }
    static __device__ __forceinline__ V join(const dfloat (&a)[2]) { return dfloat2(a[0], a[1]); }
    static __device__ __forceinline__ void split(V v, dfloat (&a)[2]) { v.split(a[0], a[1]); }
    static __device__ __forceinline__ V right(V v) {
        dfloat a, b;
        v.split(a, b);
        return dfloat2(b, shfl_down1(a));
    }
    static __device__ __forceinline__ V left(V v) {
        dfloat a, b;
        v.split(a, b);
        return dfloat2(shfl_up1(b), a);
    }
};
template <typename T> struct LaneAcc { typedef typename Acc<T>::type type; };
template <> struct LaneAcc<dfloat> { typedef DFAcc2 type; };

// strips of an nx x ny grid: across (w columns), and down in rows of h
template <typename T> __host__ __device__ constexpr int strip_width() { return 32 * Lane<T>::N - 2; }
__host__ __device__ inline int strips_across(int nx, int w) { return (nx + w - 1) / w; }
__host__ __device__ inline int strips_down(int ny, int h) { return (ny + h - 1) / h; }

// March strip (sx, sy) of height h.  At a node's offset g (32 bits: operators have fewer than
// 2^31 nodes): load(g, q, n) loads what the stencil input u is made of (q is of type Q, one
// for each column n of the lane); make_u(q) forms u; put_u(g, u) stores what belongs to an owned
// node; load2(g, q2, n) and node(q2, u, y, g, on) do the same for the outputs, y = A u, with
// on[n] telling which of the lane's columns are owned (the values of the others are
// arbitrary).  Loads run one row ahead (without that for
// the planes a double-float iteration at 2049x1025 took 128 us where it took 122 with, as kernels a phase);
// addresses out of the grid are clamped, since no owned node uses a value from there.
template <typename T, bool CROSS, bool HC, class Q, class Q2, class Load, class MakeU, class PutU, class Load2, class Node>
__device__ __forceinline__ void march_strip(const Op2D<T> &op, int sx, int sy, int h, Load load, MakeU make_u,
                                            PutU put_u, Load2 load2, Node node) {
    typedef Lane<T> LN;
    typedef typename LN::V V;
    constexpr int N = LN::N;
    const int nx = op.nx, ny = op.ny, lane = threadIdx.x & 31;
    const int j0 = sy * h, j1 = j0 + h < ny ? j0 + h : ny;         // rows j0 .. j1-1
    unsigned gi[N], ci[N];
    bool on[N];
#pragma unroll
    for (int n = 0; n < N; ++n) {
        const int q = lane * N + n, i = sx * strip_width<T>() - 1 + q;    // node column; the cell to its right is i + 1
        gi[n] = i < 0 ? i + nx - 1 : i < nx ? i : i == nx ? 1 : 0;        // periodic with the duplicated seam
        ci[n] = i + 1 <= nx ? i + 1 : nx;
        on[n] = q >= 1 && q <= strip_width<T>() && i < nx;
    }
    auto row = [&](int j) {                            // node row j; past the strip's last one, that one again
        if (j < 0) return (unsigned)(op.ymirror ? 1 : ny - 2);            // mirror (LAMB_BDRY) or wrap
        if (j > j1) j = j1;
        if (j == ny) return (unsigned)(op.ymirror ? ny - 2 : 1);
        return (unsigned)j;
    };
    Q qa[N], qb[N];
    Q2 na[N], nb[N];
    T da[N], db[N], ha[N], hb[N];
    T cb[N][4], ca[N][4];
    auto fetch_u = [&](int j, Q (&q)[N]) {
        const unsigned r = row(j) * (unsigned)nx;
#pragma unroll
        for (int n = 0; n < N; ++n) load(r + gi[n], q[n]);
    };
    auto fetch_cell = [&](int j) {                     // cell row j, between node rows j-1 and j
        const unsigned r = (unsigned)(j < j1 ? j : j1) * (unsigned)(nx + 1);
#pragma unroll
        for (int n = 0; n < N; ++n) {
            cb[n][0] = op.axx[r + ci[n]];
            cb[n][1] = op.ayy[r + ci[n]];
            if (CROSS) {
                cb[n][2] = op.axy[r + ci[n]];
                cb[n][3] = op.ayx[r + ci[n]];
            }
        }
    };
    auto fetch_node = [&](int j) {
        const unsigned r = (unsigned)(j < j1 - 1 ? j : j1 - 1) * (unsigned)nx;
#pragma unroll
        for (int n = 0; n < N; ++n) {
            load2(r + gi[n], nb[n]);
            db[n] = op.dinv[r + gi[n]];
            if (HC) hb[n] = op.hc[r + gi[n]];
        }
    };
    auto plane = [&](const T (&a)[N][4], int k) {
        T t[N];
#pragma unroll
        for (int n = 0; n < N; ++n) t[n] = a[n][k];
        return LN::join(t);
    };
    fetch_u(j0 - 1, qa);
    fetch_u(j0, qb);
    fetch_cell(j0);
    fetch_node(j0);
    V up = make_u(qa), upr = LN::right(up), mprev = up, plprev = up;    // row j-1: u and its right neighbour; cell row j-1: M, left P
    for (int j = j0; j <= j1; ++j) {                   // u of row j, cell row j, node row j-1
#pragma unroll
        for (int n = 0; n < N; ++n) {
            qa[n] = qb[n];
            na[n] = nb[n];
            da[n] = db[n];
            if (HC) ha[n] = hb[n];
#pragma unroll
            for (int k = 0; k < (CROSS ? 4 : 2); ++k) ca[n][k] = cb[n][k];
        }
        fetch_u(j + 1, qb);
        fetch_cell(j + 1);
        fetch_node(j);
        const V u = make_u(qa), ur = LN::right(u);
        if (j < j1) {
            T t[N];
            LN::split(u, t);
#pragma unroll
            for (int n = 0; n < N; ++n)
                if (on[n]) put_u((unsigned)j * (unsigned)nx + gi[n], t[n]);
        }
        const V d1 = ur - up, d2 = upr - u;            // BR - TL, TR - BL
        const V gx = d1 + d2, gy = d1 - d2;            // twice the cell's differences: the planes hold the half
        V fx = plane(ca, 0) * gx, fy = plane(ca, 1) * gy;
        if (CROSS) {
            fx = fx + plane(ca, 2) * gy;
            fy = fy + plane(ca, 3) * gx;
        }
        const V P = fx + fy, M = fx - fy, pl = LN::left(P), ml = LN::left(M);
        if (j > j0) {
            // node row j-1: TR and TL in the cell row above it, BL and BR in this one
            V s = (mprev - ml) + (P - plprev);
            if (HC) s = s + LN::join(ha) * up;
            unsigned g[N];
#pragma unroll
            for (int n = 0; n < N; ++n) g[n] = (unsigned)(j - 1) * (unsigned)nx + gi[n];
            node(na, up, s * LN::join(da), g, on);
        }
        mprev = M;
        plprev = pl;
        up = u;
        upr = ur;
    }
}

// Rows per strip.  A strip costs h + 2 rows (its own and the neighbours') of its SM quarter's
// arithmetic, the quarter with the most strips takes them one after the other, and every turn
// of the resident warps waits for one strip's latency besides, LAT tenths of a row's
// arithmetic (a row: FP64 17 operations of 65 clocks, double-float 254 of 2, FP32 some 70 in
// all).  Measured, us a BiCGStab iteration at h rows (* what the rule takes):
//   2049x1025 double-float  8: 102, 12: 109, 16: 99, 20: 98, 24: 106, 30: 107, 40: 121, rule: 97*
//   2049x1025 FP64          8: 184, 12: 183, 16: 179, 20: 181, 24: 198, 30: 175, 40: 176, rule: 175*
//   161x81 FP64             1: 23.0, 2: 21.3*, 3: 22.2, 4: 26.2, 8: 30.3
//   161x81 double-float     1: 23.5, 2: 26.6*, 3: 27.0, 4: 28.1, 8: 31.9
// Two rows at least: one is slower in FP64.  Double-float would gain from one row, but another height
// is another order of the sums, and a solve of hundreds of iterations then ends elsewhere within its
// tolerance: with one row a 161x81 projection (test_gpu_projection.py, df64-none-full) is 1.6e-8 from
// the reference's momenta, whose limit there is 1e-8.
template <typename T> struct StripLat { static constexpr int tenths = 140; };
template <> struct StripLat<double> { static constexpr int tenths = 5; };
template <> struct StripLat<dfloat> { static constexpr int tenths = 15; };

// strips(h): the strips of all grids at height h
template <typename T, class Strips>
inline int best_strip_height(Strips strips_at, int sms, int warps_per_sm) {
    const long long quarters = 4LL * sms, warps = (long long)sms * warps_per_sm;
    int best = 2;
    long long best_cost = -1;
    for (int h = 2; h <= 64; ++h) {
        const long long strips = strips_at(h);
        const long long cost = (h + 2) * (10 * ((strips + quarters - 1) / quarters) +
                                          StripLat<T>::tenths * ((strips + warps - 1) / warps));
        if (best_cost < 0 || cost < best_cost) {
            best_cost = cost;
            best = h;
        }
    }
    return best;
}

template <typename T>
inline int strip_height(int nx, int ny, int sms, int warps_per_sm) {
    const long long across = strips_across(nx, strip_width<T>());
    return best_strip_height<T>([&](int h) { return across * strips_down(ny, h); }, sms, warps_per_sm);
}

}  // namespace bella
