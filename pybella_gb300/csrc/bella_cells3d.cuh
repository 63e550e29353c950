// bella_cells3d.cuh -- what the 3D projection (bella_proj3d.cu) and its explicit parts
// (bella_expl3d.cu) share on the device: the launch shape of the kernels that walk along
// x with a (y, z) tile, the nodal divergence, the 2x2x2 pressure gradient of a plane
// pair, and the implicit Coriolis / buoyancy factors.
//
// These kernels are bound by GB300's FP64 pipe (about two lanes per SM and clock), not by
// memory: what counts is FP64 operations per cell, an IEEE division being about ten and
// pow more than a hundred.  So divisions by grid constants become products with
// reciprocals formed once on the host, sums over 2x2x2 cells are built from the sums of
// two planes, of which the walk keeps one, and a cell's quotients are formed once per cell.
#pragma once
#include "bella_internal.cuh"

namespace bella {

constexpr int C3_K = 32, C3_J = 8;      // tile of a block: C3_K along z (a warp's row), C3_J along y
constexpr int C3_THREADS = C3_K * C3_J;

struct Walk3 {
    int seg;                            // planes along x per block
    TileRow tiles;                      // z, y and the segments
};

// Blocks of ny x nz tiles, walking nx planes in equal segments that each read `extra`
// more planes: the number of segments with the least work on the fullest SM.
inline Walk3 walk3(int nx, int ny, int nz, int extra) {
    Walk3 w;
    const int ty = (ny + C3_J - 1) / C3_J, tz = (nz + C3_K - 1) / C3_K;
    const long long tiles = (long long)ty * tz, sms = num_sms();
    long long best = -1;
    w.seg = nx;
    for (int n = 1; n <= 16 && n <= nx; ++n) {
        const int seg = (nx + n - 1) / n;
        const long long cost = ((tiles * ((nx + seg - 1) / seg) + sms - 1) / sms) * (seg + extra);
        if (best < 0 || cost < best) {
            best = cost;
            w.seg = seg;
        }
    }
    w.tiles = tile_row(tz, ty, (nx + w.seg - 1) / w.seg);
    return w;
}

// sums of a node plane's four nodes around a cell of row (j, k): x, y and z parts of
// grad_nodes (second_projection.py:496-521); the gradient of a cell is
// (b.x - a.x, a.y + b.y, a.z + b.z) over its two planes, times 0.25 / spacing
struct PlaneGrad { double x, y, z; };

__device__ __forceinline__ PlaneGrad plane_grad(const double *p, long long n, int ncz) {
    const double p00 = p[n], p01 = p[n + 1], p10 = p[n + ncz], p11 = p[n + ncz + 1];
    const double a = p00 + p01, b = p10 + p11;
    PlaneGrad g;
    g.x = a + b;
    g.y = b - a;
    g.z = (p01 - p00) + (p11 - p10);
    return g;
}

// the factors of multiply_inverse_coriolis (second_projection.py:604-646) with what does
// not depend on the cell formed once: cor_coef's entries are affine in nu + nonhydro
struct Coriolis3 {
    double nh, wh1, wv, wh2;
    double uu0, uv, uwh, vu, vv, vw, wuh, wvv, ww0, d0, d1;   // see cor_matrix
    int on;                                                   // any Coriolis component
};

inline Coriolis3 coriolis3(double dt, double nonhydro, const double *cor) {
    Coriolis3 c;
    c.nh = nonhydro;
    c.wh1 = dt * cor[0]; c.wv = dt * cor[1]; c.wh2 = dt * cor[2];
    c.uu0 = c.wh1 * c.wh1;
    c.uv = nonhydro * (c.wh1 * c.wv + c.wh2);
    c.uwh = c.wh1 * c.wh2;
    c.vu = c.wh1 * c.wv - c.wh2;
    c.vv = nonhydro * (1.0 + c.wv * c.wv);
    c.vw = c.wh2 * c.wv + c.wh1;
    c.wuh = c.wh1 * c.wh2;
    c.wvv = nonhydro * (c.wh2 * c.wv - c.wh1);
    c.ww0 = c.wh2 * c.wh2;
    c.d0 = c.wh1 * c.wh1 + c.wh2 * c.wh2;
    c.d1 = c.wv * c.wv + 1.0;
    c.on = c.wh1 != 0.0 || c.wv != 0.0 || c.wh2 != 0.0;
    return c;
}

// neither zero nor below the normal numbers nor infinite nor NaN
__device__ __forceinline__ bool is_normal(double v) {
    return (unsigned)((__double2hiint(v) & 0x7fffffff) - 0x00100000) < 0x7fe00000u;
}
__device__ __forceinline__ bool are_finite(double a, double b, double c) {
    const int x = __double2hiint(a) & 0x7fffffff, y = __double2hiint(b) & 0x7fffffff, z = __double2hiint(c) & 0x7fffffff;
    return max(max(x, y), z) < 0x7ff00000;
}

// Without Coriolis forces the inverse of (u, v, w) is diag(1, nonhydro / q, 1) with q = nu + nonhydro =
// qr / rho.  Not where one of the three or qr is not finite, or qr is zero: there the whole formula
// stands, in which each component enters the others times zero and hands them its NaN.
__device__ __forceinline__ bool cor_diagonal(const Coriolis3 &c, double qr, double u, double v, double w) {
    return !c.on && is_normal(qr) && are_finite(u, v, w);
}

// (U, V, W) <- the inverse applied to them
__device__ __forceinline__ void cor_apply(const Coriolis3 &c, double q, double &U, double &V, double &W) {
    const double den = 1.0 / (c.d0 + q * c.d1);
    const double u = (c.uu0 + q) * U + c.uv * V + (c.uwh - q * c.wv) * W;
    const double v = c.vu * U + c.vv * V + c.vw * W;
    const double w = (c.wuh + q * c.wv) * U + c.wvv * V + (q + c.ww0) * W;
    U = den * u; V = den * v; W = den * w;
}

// scale_wall_node_values (second_projection.py:433-474) is 1 off the first and last two
// inner node rows of the wall axes
template <class G>
__device__ __forceinline__ double node_wall_scale(const G &P, int a, int b, int c, double f) {
    const int n[3] = {P.icx - 1, P.icy - 1, P.icz - 1}, x[3] = {a, b, c};
    bool near = false;
#pragma unroll
    for (int d = 0; d < 3; ++d) near = near || (P.bc[d] && (x[d] == 1 || x[d] == n[d] - 2));
    if (!near) return 1.0;
    int wall[3], nn[3], xx[3];
#pragma unroll
    for (int d = 0; d < 3; ++d) { wall[d] = P.bc[d]; nn[d] = n[d]; xx[d] = x[d]; }
    return wall_scale(3, xx, nn, wall, f);
}

// divergence_nodes' 3D branch (second_projection.py:556-570) on node.isc for both its
// callers: op(a, b, c, div, s) gets the divergence and, with POW, the 2x2x2 sum of
// weighted_pow(rhoY, expo, weight).  cx, cy, cz: 0.25 / spacing, cx with the sign of the x term.  A block
// walks an 8x32 tile of nodes along x; the momenta weighted with Y of a plane's 9x33
// cells go through shared memory (one division each), each node keeps its last plane's
// sums.
template <bool POW, class G, class Op>
__device__ __forceinline__ void walk_divergence(const G &P, const Walk3 &walk, const double *rho, const double *rhou,
                                                const double *rhov, const double *rhow, const double *rhoY, double cx,
                                                double cy, double cz, double expo, double weight, Op op) {
    constexpr int NJ = C3_J + 1, NK = C3_K + 1, NE = NJ * NK;
    __shared__ double sm[2][POW ? 4 : 3][NE];
    const int t = threadIdx.x, tk = t % C3_K, tj = t / C3_K;
    const uint3 tile = tile_of(walk.tiles);
    const int k0 = tile.x * C3_K, j0 = tile.y * C3_J;
    const int a0 = tile.z * walk.seg, a1 = a0 + walk.seg < P.icx - 1 ? a0 + walk.seg : P.icx - 1;    // nodes a0 .. a1-1
    const int b = j0 + tj, c = k0 + tk;
    const bool on = b < P.icy - 1 && c < P.icz - 1;
    const long long plane = (long long)P.icy * P.icz;
    double U1 = 0.0, V1 = 0.0, W1 = 0.0, S1 = 0.0;
    int buf = 0;
    for (int p = a0; p <= a1; ++p, buf ^= 1) {
        for (int e = t; e < NE; e += C3_THREADS) {
            const int lj = e / NK, lk = e - lj * NK, gj = j0 + lj, gk = k0 + lk;
            if (gj < P.icy && gk < P.icz) {
                const long long x = p * plane + (long long)gj * P.icz + gk;
                const double rY = rhoY[x], Y = rY / rho[x];
                sm[buf][0][e] = rhou[x] * Y;
                sm[buf][1][e] = rhov[x] * Y;
                sm[buf][2][e] = rhow[x] * Y;
                if (POW) sm[buf][3][e] = weighted_pow(rY, expo, weight);
            }
        }
        __syncthreads();                                // the other buffer's readers are past it
        const int e = tj * NK + tk;
        const double *u = sm[buf][0], *v = sm[buf][1], *w = sm[buf][2];
        const double U = (u[e] + u[e + 1]) + (u[e + NK] + u[e + NK + 1]);
        const double V = (v[e + NK] + v[e + NK + 1]) - (v[e] + v[e + 1]);
        const double W = (w[e + 1] - w[e]) + (w[e + NK + 1] - w[e + NK]);
        double S = 0.0;
        if (POW) {
            const double *q = sm[buf][3];
            S = (q[e] + q[e + 1]) + (q[e + NK] + q[e + NK + 1]);
        }
        if (on && p > a0) op(p - 1, b, c, cx * (U - U1) + cy * (V1 + V) + cz * (W1 + W), S1 + S);
        U1 = U; V1 = V; W1 = W; S1 = S;
    }
}

}  // namespace bella
