// bella_advect.cu -- the advection of the reference (explicit.py, recovery.py,
// numerical_flux.py) on the device, 2D and 3D: face mass fluxes, the Strang-split
// sweeps of advect and the first-order advect_rk.
//
// bella_advect.cuh states the arithmetic one face, cell or line at a time, operation
// by operation as the reference has it (checked on the CPU by
// tests/test_advect_host.py).  The kernels here evaluate the same formulas over
// lines and planes of cells, so that what neighbouring faces share is computed once:
//   k_adv_bd       boundary data along one axis, a thread per line and side
//   k_adv_sweep    one sweep: boundary data, fluxes, update, boundary data of whole
//                  lines; or the fluxes alone (advect_rk)
//   k_adv_update   advect_rk's update by the fluxes of all axes, with its pwchi
//   k_adv_mass2/3  the face mass fluxes of all axes in one pass
// What bounds them is GB300's FP64 pipe (about two lanes per SM and clock), so the
// measure of these kernels is FP64 operations per cell: an IEEE division is about
// ten.  One thread per face with the formulas as they stand took 54 divisions a face
// (8.45 ms per 3D sweep at 257x129x257 nodes, with 0.87 ms for its update) and 18 a
// face for the mass fluxes (2.9 ms per axis).
#include "bella_advect.cuh"
#include "bella_internal.cuh"

namespace bella {

constexpr int SW_THREADS = 256;

// The lines of a sweep along axis s: cell c of line (o, k) at o*so + k*sk + c*sc, its
// face f at face_line(o, k)*(ns+1) + f.  Threads run along k (unit stride) when the sweep
// axis is not the contiguous one, along c when it is.  (k, o) are the other two
// coordinates, or k = a*n2 + b where one index covers both.
struct SweepLines {
    int s, ns, nk, no, bc;
    int n1, n2;                // extents of a and b (o and k); n1 = 0: k alone (2D)
    long long so, sk, sc, fo, fk;
};

inline SweepLines sweep_lines(const AdvGeom &G, int s) {
    SweepLines W;
    W.s = s;
    W.ns = G.ic[s];
    W.bc = G.bc[s];
    W.no = 1;
    W.so = W.fo = 0;
    W.fk = 1;
    const int last = G.nd - 1;
    if (s == last) {                                   // contiguous lines
        W.nk = G.nd == 2 ? G.ic[0] : G.ic[0] * G.ic[1];
        W.sk = G.ic[last];
        W.sc = 1;
    } else if (s == 0) {
        W.nk = G.nd == 2 ? G.ic[1] : G.ic[1] * G.ic[2];
        W.sk = 1;
        W.sc = W.nk;
    } else {                                           // y in 3D: faces ordered (z, x, y)
        W.nk = G.ic[2];
        W.no = G.ic[0];
        W.so = (long long)G.ic[1] * G.ic[2];
        W.sk = 1;
        W.sc = G.ic[2];
        W.fk = G.ic[0];
        W.fo = 1;
    }
    W.n1 = G.nd == 2 ? 0 : G.ic[s == 0 ? 1 : 0];
    W.n2 = G.nd == 2 ? W.nk : G.ic[s == 2 ? 1 : 2];
    return W;
}

// boundary data of one end of a line (adv_bd_line's two ghost cells of that side): side 0
// the low end.  The ghost cells of one side read inner cells and each other, never
// the other side's.
__device__ __forceinline__ void bd_side(const AdvGeom &G, const SweepLines &W, const AdvFields &F, long long base,
                                        int side, const double *rhoY0, const double *strat_inv) {
    const int n = W.ns;
    auto at = [&](int c) { return base + c * W.sc; };
    if (W.s != 1 || G.g == 0.0) {
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            double *a = F.f[q];
            if (W.bc == 0) {
                const double v0 = a[at(side ? 2 : n - 4)], v1 = a[at(side ? 3 : n - 3)];
                a[at(side ? n - 2 : 0)] = v0;
                a[at(side ? n - 1 : 1)] = v1;
            } else if (q != 3) {
                const double sg = (q == 2) ? -1.0 : 1.0;
                const double v0 = a[at(side ? n - 3 : 2)], v1 = a[at(side ? n - 4 : 3)];
                a[at(side ? n - 2 : 1)] = sg * v0;
                a[at(side ? n - 1 : 0)] = sg * v1;
            }
        }
        return;
    }
    const double gm1 = G.gamm - 1.0;
    const double dir = side ? -1.0 : 1.0;
#pragma unroll
    for (int cur = 1; cur >= 0; --cur) {
        const int ci = side ? n - 1 - cur : cur;                     // ghost cell
        const long long S_ = at(side ? n - 4 + cur : 3 - cur);       // its mirror image
        const long long I = at(ci);
        const double rs = F.f[0][S_], inv = 1.0 / rs;
        const double image = -F.f[2][S_] * F.f[4][S_] * inv;
        const double S = strat_inv[ci];
        double rY;
        if (G.is_compressible == 1) {
            const long long L = at(side ? ci - 1 : ci + 1);
            const double rl = F.f[4][L], Y_last = rl / F.f[0][L];
            const double dpi = dir * (gm1 / G.gamm * G.g) * 0.5 * G.d[1] * (1.0 / Y_last + S);
            rY = pow(pow(rl, gm1) + dpi, 1.0 / gm1);
        } else {
            rY = rhoY0[ci];
        }
        const double r = rY * S;
        const double u = F.f[1][S_] * inv, w = F.f[3][S_] * inv, X = F.f[5][S_] * inv;
        F.f[0][I] = r;
        F.f[1][I] = r * u;
        F.f[2][I] = r * (image / rY);
        F.f[3][I] = r * w;
        F.f[4][I] = rY;
        F.f[5][I] = r * X;
    }
}

// boundary data along one axis, for the advection and for the projections and their explicit
// parts: two threads per line and an IEEE division fewer per quantity than a thread per line
// working both ends in turn (boundary.py:56-132 as it stands): 19.6 -> 7.0 us at 161x81
// nodes, along y at 257x129x257 42 -> 15 us (ncu)
__global__ void __launch_bounds__(128) k_adv_bd(AdvGeom G, SweepLines W, AdvFields F, const double *rhoY0, const double *strat_inv) {
    dependents_may_start();
    wait_for_previous();
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x, nl = (long long)W.no * W.nk;
    if (e >= 2 * nl) return;
    const int side = e >= nl ? 1 : 0;
    const long long l = e - side * nl;
    const int o = (int)(l / W.nk), k = (int)(l - (long long)o * W.nk);
    bd_side(G, W, F, o * W.so + k * W.sk, side, rhoY0, strat_inv);
}

__device__ __forceinline__ bool not_finite(double v) { return (__double2hiint(v) & 0x7ff00000) == 0x7ff00000; }

// One sweep of whole lines (explicit_step_and_flux, explicit.py:77-158): boundary data
// along the axis, the upwind fluxes of every inner face, the conservative update in
// place, boundary data again.  FLUX_ONLY (advect_rk): boundary data and fluxes with
// lambda 0 in the recovery.
//
// A block takes L lines from end to end in chunks of C = 256/L cells, one thread
// per (cell, line), in three stages with a block barrier between them: the cells'
// primitives into shared memory; the flux of face c-1 from the cells c-3 .. c; the
// update of cell c-2 from its two faces.  Lines are owned by one block, so the update
// can be in place.  Per cell and sweep that is two divisions and about 50 FP64
// operations: u = rhou (1/rho) and so on; the recovered state enters the flux as q and
// 1/Y, which get_conservatives and primitives (recovery.py:241-262) leave unchanged up
// to rounding (q rho / rho); and of the two states of a face only the upwind one is
// evaluated, unless a cell in reach is not finite (then both are, as the weights 0 and
// 1 of the other side keep a NaN).
// L: 32 lines (a warp's unit-stride row) where that fills the chip, else 4, else 1, and 8
// or 1 contiguous lines (DevEx::sweep); C*L threads always hold one cell each.
// Measured (GB300, ncu; 257x129x257 nodes, 8.9 M cells): 0.88 to 0.95 ms a sweep with its update along
// x and y, 0.89 along z (8.45 + 0.87 before), the fluxes alone 0.60 to 0.65 ms; at 161x81
// 11.5 and 12.4 us (42 + 6.7 before, with 2 x 20 us of boundary data).  The FP64 pipe takes 47 to 54
// instructions a cell and sweep (sm__inst_executed_pipe_fp64), for the fluxes alone 32 to 37; at the
// 0.505e12 a second of an FMA chain that is 0.83 to 0.96 ms: it runs at the pipe's rate.
template <int L, bool CONTIG, bool FLUX_ONLY>
__global__ void __launch_bounds__(SW_THREADS, 3)
k_adv_sweep(AdvGeom G, SweepLines W, AdvFields F, double lmbda, AdvFaces out, int write_faces, const double *rhoY0,
            const double *strat_inv) {
    dependents_may_start();
    wait_for_previous();
    constexpr int C = SW_THREADS / L;
    constexpr int R = C + 4;                           // ring of cells: a chunk and the three before it
    __shared__ double P[5][R * L];                     // u, v, w, X, 1/Y
    __shared__ double RY[FLUX_ONLY ? 1 : R * L];       // 1/rhoY
    __shared__ double M[R * L];                        // face mass flux
    __shared__ double FL[FLUX_ONLY ? 5 : 6][R * L];    // fluxes of rho, rhou, rhov, rhow, rhoX, rhoY
    __shared__ unsigned char bad[R * L];               // a primitive of the cell is not finite

    const int ns = W.ns, t = threadIdx.x;
    const int nkb = (W.nk + L - 1) / L;
    const int o = blockIdx.x / nkb, k0 = (blockIdx.x - o * nkb) * L;
    const int tl = CONTIG ? t / C : t % L, tc = CONTIG ? t % C : t / L;
    const int fl = t / C, fc = t % C;                  // face-major mapping: consecutive faces of a line
    const bool live = k0 + tl < W.nk, flive = k0 + fl < W.nk;
    const long long base = o * W.so + (k0 + tl) * W.sk;
    const long long frow = (o * W.fo + (k0 + tl) * W.fk) * (ns + 1);
    const long long fmap = (o * W.fo + (k0 + fl) * W.fk) * (ns + 1);
    // ring slot of position p of line l
    auto at = [](int slot, int l) { return CONTIG ? l * R + slot : slot * L + l; };
    auto wrap = [](int slot) { return slot < 0 ? slot + R : slot >= R ? slot - R : slot; };

    bool inner;                                        // line off the outer ghost layer (recovery.py:60-62)
    {
        const int k = k0 + tl, a = W.no > 1 ? o : k / W.n2, b = W.no > 1 ? k : k - a * W.n2;
        inner = (W.n1 == 0 || (a >= 1 && a <= W.n1 - 2)) && b >= 1 && b <= W.n2 - 2;
    }

    if (t < 2 * L && k0 + t % L < W.nk)
        bd_side(G, W, F, o * W.so + (k0 + t % L) * W.sk, t / L, rhoY0, strat_inv);
    __syncthreads();

    double v[6], mf = 0.0;
#pragma unroll
    for (int q = 0; q < 6; ++q) v[q] = 1.0;
    auto fetch = [&](int b0) {
        if (live && b0 + tc < ns) {
            const long long e = base + (b0 + tc) * W.sc;
#pragma unroll
            for (int q = 0; q < 6; ++q) v[q] = F.f[q][e];
        }
        if (flive && b0 + fc <= ns) mf = out.f[4][fmap + b0 + fc];
    };
    fetch(0);
    int slot = tc, slot0 = 0;                          // ring slots of cell c and of the chunk's first cell
    for (int b0 = 0; b0 < ns + 2; b0 += C) {
        const int c = b0 + tc;
        if (c < ns) {                                  // 1. primitives (variable.py:56-86)
            const double ri = v[0] != 0.0 ? 1.0 / v[0] : 0.0, ryi = 1.0 / v[4];
            const double p0 = v[1] * ri, p1 = v[2] * ri, p2 = v[3] * ri, p3 = v[5] * ri;
            const double p4 = v[0] != 0.0 ? v[0] * ryi : INFINITY;
            const int i = at(slot, tl);
            P[0][i] = p0; P[1][i] = p1; P[2][i] = p2; P[3][i] = p3; P[4][i] = p4;
            if (!FLUX_ONLY) RY[i] = ryi;
            bad[i] = not_finite(p0) || not_finite(p1) || not_finite(p2) || not_finite(p3) || not_finite(p4);
        }
        M[at(wrap(slot0 + fc), fl)] = mf;
        fetch(b0 + C);
        __syncthreads();
        const int f = c - 1;
        if (live && f >= 0 && f <= ns) {               // 2. flux of face f, between cells f-1 and f
            const int sf = wrap(slot - 1), i0 = at(sf, tl);
            const double m = M[i0];
            double x[5];                               // rho, rhou, rhov, rhow, rhoX
            if (f == 0 || f == ns) {
                const int qs[5] = {0, 1, 2, 3, 5};
#pragma unroll
                for (int q = 0; q < 5; ++q) x[q] = out.f[qs[q]][frow + f];
            } else {
                // state of cell a (ring slot sa) at its right (sgn 1) or left (sgn -1) face
                auto side = [&](int a, int sa, double sgn, double *y) {
                    const int i = at(sa, tl);
                    double w = 0.0;
                    int ip = i, im = i;
                    if (a >= 1 && a <= ns - 2) {       // the slope of the first and last cell is zero
                        ip = at(wrap(sa + 1), tl);
                        im = at(wrap(sa - 1), tl);
                        w = 0.25 * sgn;                // half the cell, mean of the two differences
                        if (!FLUX_ONLY && inner) w = fma(-0.125 * lmbda * (M[i] + M[ip]), RY[i], w);
                    }
#pragma unroll
                    for (int q = 0; q < 5; ++q) y[q] = fma(w, P[q][ip] - P[q][im], P[q][i]);
                };
                const int sl = wrap(slot - 2);
                const double ml = M[at(sl, tl)], mr = M[at(slot, tl)];
                const int b = not_finite(m) | not_finite(ml) | not_finite(mr) | bad[i0] | bad[at(sl, tl)] | (f >= 2 ? bad[at(wrap(slot - 3), tl)] : 0) |
                              (f + 1 < ns ? bad[at(slot, tl)] : 0);
                const bool up = m > 0.0;
                double y[5];
                if (!b) {
                    side(up ? f - 1 : f, up ? sl : sf, up ? 1.0 : -1.0, y);
                    const double g = m * y[4];
                    x[0] = g;
#pragma unroll
                    for (int q = 0; q < 4; ++q) x[q + 1] = g * y[q];
                } else {
                    double z[5];
                    side(f - 1, sl, 1.0, y);
                    side(f, sf, -1.0, z);
                    const double a0 = (up ? 1.0 : m < 0.0 ? 0.0 : 0.5) * y[4];
                    const double a1 = (up ? 0.0 : m < 0.0 ? 1.0 : 0.5) * z[4];
                    // the face density (recovery.py:117-119) cancels while it and Y are finite
                    // and the cells' velocities (recovery.py:60-62) weigh their slopes
                    double den = P[W.s][at(sl, tl)] + P[W.s][i0] + y[4] + z[4];
                    if (inner && f - 1 >= 1) den += 0.0 * (ml + m);
                    if (inner && f <= ns - 2) den += 0.0 * (m + mr);
                    const double keep = not_finite(den) ? NAN : 1.0;
                    x[0] = keep * m * (a0 + a1);
#pragma unroll
                    for (int q = 0; q < 4; ++q) x[q + 1] = keep * m * (a0 * y[q] + a1 * z[q]);
                }
            }
#pragma unroll
            for (int q = 0; q < 5; ++q) FL[q][i0] = x[q];
            if (!FLUX_ONLY) FL[5][i0] = m;             // M's slot is refilled while the update reads
        }
        __syncthreads();
        const int e = c - 2;
        if (!FLUX_ONLY && live && e >= 0 && e < ns) {  // 3. update of cell e (explicit.py:146-151)
            const int ia = at(wrap(slot - 2), tl), ib = at(wrap(slot - 1), tl);
            const long long g = base + e * W.sc;
            const int qs[5] = {0, 1, 2, 3, 5};
            double old[6];
#pragma unroll
            for (int q = 0; q < 6; ++q) old[q] = F.f[q][g];
#pragma unroll
            for (int q = 0; q < 5; ++q) F.f[qs[q]][g] = old[qs[q]] + lmbda * (FL[q][ia] - FL[q][ib]);
            F.f[4][g] = old[4] + lmbda * (FL[5][ia] - FL[5][ib]);
        }
        if (write_faces) {
            const int ff = b0 - 1 + fc;
            if (flive && ff >= 1 && ff <= ns - 1) {
                const int i = at(wrap(slot0 - 1 + fc), fl);
                const int qs[5] = {0, 1, 2, 3, 5};
#pragma unroll
                for (int q = 0; q < 5; ++q) out.f[qs[q]][fmap + ff] = FL[q][i];
            }
        }
        slot = wrap(slot + C);
        slot0 = wrap(slot0 + C);
    }
    if (FLUX_ONLY) return;
    __syncthreads();
    if (t < 2 * L && k0 + t % L < W.nk)
        bd_side(G, W, F, o * W.so + (k0 + t % L) * W.sk, t / L, rhoY0, strat_inv);
}

// advect_rk's update by the fluxes of all axes (explicit.py:222-249), in the order x, y, z, and
// its rhoX update of the y sweep.  Threads run along the contiguous axis; in 3D each takes
// UPD_X cells along x, whose x faces are consecutive: 0.74 ms at 257x129x257 (ncu), against
// 0.87 ms for each axis alone with threads along that axis's lines.
// LONG: the tiles in one row of blocks (tile_of), for extents past a grid's; the others keep their grid, with
// which the compiler unrolls the cells' loop (64 registers for 34: 0.74 ms for 0.90).
constexpr int UPD_X = 8;
template <int ND, bool LONG>
__global__ void __launch_bounds__(256)
k_adv_update(AdvGeom G, TileRow tiles, AdvFields F, AdvFaces fx, AdvFaces fy, AdvFaces fz, double lx, double ly, double lz,
             double *pw) {
    dependents_may_start();
    wait_for_previous();
    const int icx = G.ic[0], icy = G.ic[1], icz = G.ic[2];
    const uint3 tile = LONG ? tile_of(tiles) : make_uint3(blockIdx.x, blockIdx.y, blockIdx.z);
    const int k = tile.x * 32 + threadIdx.x;           // z in 3D, y in 2D
    const int r = tile.y * 8 + threadIdx.y;            // y in 3D, x in 2D
    if (k >= (ND == 3 ? icz : icy) || r >= (ND == 3 ? icy : icx)) return;
    const int i0 = ND == 3 ? (int)tile.z * UPD_X : r, i1 = ND == 3 ? (i0 + UPD_X < icx ? i0 + UPD_X : icx) : r + 1;
    const int j = ND == 3 ? r : k;
    for (int i = i0; i < i1; ++i) {
        const long long e = ND == 3 ? ((long long)i * icy + j) * icz + k : (long long)i * icy + j;
        const long long ax = (ND == 3 ? (long long)j * icz + k : (long long)j) * (icx + 1) + i;
        const long long ay = (ND == 3 ? (long long)k * icx + i : (long long)i) * (icy + 1) + j;
        const long long az = ((long long)i * icy + j) * (icz + 1) + k;
#pragma unroll
        for (int q = 0; q < 6; ++q) {
            double u = F.f[q][e] + lx * (fx.f[q][ax] - fx.f[q][ax + 1]);
            const double dy = ly * (fy.f[q][ay] - fy.f[q][ay + 1]);
            u += dy;
            if (ND == 3) u += lz * (fz.f[q][az] - fz.f[q][az + 1]);
            F.f[q][e] = u;
            if (q == 5 && pw) pw[e] = dy;
        }
    }
}

// Face mass fluxes of all axes in one pass (recompute_advective_fluxes,
// numerical_flux.py:5-46): m = rhoY mom / rho once per cell with one division,
// the weighted boxes from shared memory.  3D: a block holds an 8x32 (y, z) tile of
// the planes x = a-1 .. b and keeps the sums of the last two planes in registers.
// Outer faces are not written.  1.03 ms at 257x129x257 nodes (ncu) against 8.7 ms for the
// three axes with a thread per face and its 18 divisions.
constexpr int MS_J = 8, MS_K = 32, MS_X = 64;
template <bool LONG>                                   // as k_adv_update's
__global__ void __launch_bounds__(MS_J *MS_K)
k_adv_mass3(AdvGeom G, TileRow tiles, AdvFields F, double *mx, double *my, double *mz) {
    dependents_may_start();
    wait_for_previous();
    constexpr int NJ = MS_J + 2, NK = MS_K + 2;
    __shared__ double sm[2][3][NJ][NK];
    const int icx = G.ic[0], icy = G.ic[1], icz = G.ic[2];
    const int t = threadIdx.x, tk = t % MS_K, tj = t / MS_K;
    const uint3 tile = LONG ? tile_of(tiles) : make_uint3(blockIdx.x, blockIdx.y, blockIdx.z);
    const int k0 = 1 + tile.x * MS_K, j0 = 1 + tile.y * MS_J;
    const int a = 1 + tile.z * MS_X, b = a + MS_X < icx ? a + MS_X : icx;   // x faces a .. b-1
    const int j = j0 + tj, k = k0 + tk;                // inner cell, or the last face
    const bool in_j = j <= icy - 2, in_k = k <= icz - 2, on = j <= icy - 1 && k <= icz - 1;
    double B1 = 0.0, C1 = 0.0, C2 = 0.0, D1 = 0.0, D2 = 0.0;
    int buf = 0;
    for (int p = a - 1; p <= b && p < icx; ++p, buf ^= 1) {
        for (int e = t; e < NJ * NK; e += MS_J * MS_K) {
            const int lj = e / NK, lk = e - lj * NK, gj = j0 - 1 + lj, gk = k0 - 1 + lk;
            double m0 = 0.0, m1 = 0.0, m2 = 0.0;
            if (gj < icy && gk < icz) {
                const long long c = ((long long)p * icy + gj) * icz + gk;
                const double Y = F.f[4][c] / F.f[0][c];
                m0 = F.f[1][c] * Y; m1 = F.f[2][c] * Y; m2 = F.f[3][c] * Y;
            }
            sm[buf][0][lj][lk] = m0; sm[buf][1][lj][lk] = m1; sm[buf][2][lj][lk] = m2;
        }
        __syncthreads();                               // the other buffer's readers are past it
        double row[3], C, D;
#pragma unroll
        for (int q = 0; q < 3; ++q)
            row[q] = fma(2.0, sm[buf][0][tj + q][tk + 1], sm[buf][0][tj + q][tk] + sm[buf][0][tj + q][tk + 2]);
        const double B = fma(2.0, row[1], row[0] + row[2]);
        {
            double z[3], y[3];
#pragma unroll
            for (int q = 0; q < 3; ++q) {
                z[q] = sm[buf][1][tj][tk + q] + sm[buf][1][tj + 1][tk + q];       // cells j-1 and j
                y[q] = sm[buf][2][tj + q][tk] + sm[buf][2][tj + q][tk + 1];       // cells k-1 and k
            }
            C = fma(2.0, z[1], z[0] + z[2]);
            D = fma(2.0, y[1], y[0] + y[2]);
        }
        if (on) {
            if (p >= a && p < b && in_j && in_k) mx[((long long)j * icz + k) * (icx + 1) + p] = (B1 + B) * (1.0 / 32.0);
            const int i = p - 1;
            if (i >= a && i < b && i <= icx - 2) {
                if (in_k) my[((long long)k * icx + i) * (icy + 1) + j] = fma(2.0, C1, C2 + C) * (1.0 / 32.0);
                if (in_j) mz[((long long)i * icy + j) * (icz + 1) + k] = fma(2.0, D1, D2 + D) * (1.0 / 32.0);
            }
        }
        B1 = B;
        C2 = C1; C1 = C;
        D2 = D1; D1 = D;
    }
}

template <bool LONG>
__global__ void __launch_bounds__(256) k_adv_mass2(AdvGeom G, TileRow tiles, AdvFields F, double *mx, double *my) {
    dependents_may_start();
    wait_for_previous();
    __shared__ double sm[2][10][34];
    const int icx = G.ic[0], icy = G.ic[1];
    const int t = threadIdx.x, tj = t % 32, ti = t / 32;
    const uint3 tile = LONG ? tile_of(tiles) : make_uint3(blockIdx.x, blockIdx.y, 0);
    const int j0 = 1 + tile.x * 32, i0 = 1 + tile.y * 8;
    for (int e = t; e < 10 * 34; e += 256) {
        const int li = e / 34, lj = e - li * 34, gi = i0 - 1 + li, gj = j0 - 1 + lj;
        double m0 = 0.0, m1 = 0.0;
        if (gi < icx && gj < icy) {
            const long long c = (long long)gi * icy + gj;
            const double Y = F.f[4][c] / F.f[0][c];
            m0 = F.f[1][c] * Y; m1 = F.f[2][c] * Y;
        }
        sm[0][li][lj] = m0; sm[1][li][lj] = m1;
    }
    __syncthreads();
    const int i = i0 + ti, j = j0 + tj;
    if (i > icx - 1 || j > icy - 1) return;
    double x[3], y[3];
#pragma unroll
    for (int q = 0; q < 3; ++q) {
        x[q] = sm[0][ti][tj + q] + sm[0][ti + 1][tj + q];              // cells i-1 and i
        y[q] = sm[1][ti + q][tj] + sm[1][ti + q][tj + 1];              // cells j-1 and j
    }
    if (j <= icy - 2) mx[(long long)j * (icx + 1) + i] = fma(2.0, x[1], x[0] + x[2]) * 0.125;
    if (i <= icx - 2) my[(long long)i * (icy + 1) + j] = fma(2.0, y[1], y[0] + y[2]) * 0.125;
}

void adv_boundary(const AdvGeom &G, int s, const AdvFields &F, const double *rhoY0, const double *strat_inv,
                  cudaStream_t st) {
    const SweepLines W = sweep_lines(G, s);
    const long long n = 2LL * W.no * W.nk;
    launch_dependent(k_adv_bd, (unsigned)((n + 127) / 128), 128, 0, st, G, W, F, rhoY0, strat_inv);
}

namespace {

struct DevEx {
    AdvGeom G;
    AdvFields F;
    AdvFaces fl[3];
    const double *rhoY0, *strat_inv;
    double *pw;
    cudaStream_t st;

    void bd(int s) { adv_boundary(G, s, F, rhoY0, strat_inv, st); }
    // a range of tiles as a grid where its extents are within one's, else in one row (the kernels' LONG)
    static bool fits(const TileRow &t) { return t.ny <= 65535 && t.blocks / (t.nx * t.ny) <= 65535; }
    static dim3 grid_of(const TileRow &t) { return fits(t) ? dim3(t.nx, t.ny, t.blocks / (t.nx * t.ny)) : dim3(t.blocks); }
    template <int L, bool CONTIG, bool FLUX_ONLY>
    void launch(const SweepLines &W, double lmbda, int write_faces) {
        const int grid = W.no * ((W.nk + L - 1) / L);
        launch_dependent(k_adv_sweep<L, CONTIG, FLUX_ONLY>, grid, SW_THREADS, 0, st, G, W, F, lmbda, fl[W.s], write_faces,
                         rhoY0, strat_inv);
    }
    // the sweep of axis s, or its fluxes alone.  Many lines per block make full rows and few
    // barriers per cell; the line count has to leave two blocks per SM, since the FP64
    // pipe of an SM without a block is lost
    template <bool FLUX_ONLY>
    void sweep(int s, double lmbda, int write_faces) {
        const SweepLines W = sweep_lines(G, s);
        const long long lines = (long long)W.no * W.nk, full = 2LL * num_sms();
        if (s == G.nd - 1) {
            if (lines >= 8 * full) launch<8, true, FLUX_ONLY>(W, lmbda, write_faces);
            else launch<1, true, FLUX_ONLY>(W, lmbda, write_faces);
        } else if (lines >= 32 * full && W.nk >= 32) {
            launch<32, false, FLUX_ONLY>(W, lmbda, write_faces);
        } else if (lines >= 4 * full) {
            launch<4, false, FLUX_ONLY>(W, lmbda, write_faces);
        } else {
            launch<1, false, FLUX_ONLY>(W, lmbda, write_faces);
        }
    }
    void mass() {
        if (G.nd == 3) {
            const TileRow g = tile_row((G.ic[2] - 1 + MS_K - 1) / MS_K, (G.ic[1] - 1 + MS_J - 1) / MS_J,
                                       (G.ic[0] - 1 + MS_X - 1) / MS_X);
            launch_dependent(fits(g) ? k_adv_mass3<false> : k_adv_mass3<true>, grid_of(g), MS_J * MS_K, 0, st, G, g, F, fl[0].f[4], fl[1].f[4], fl[2].f[4]);
        } else {
            const TileRow g = tile_row((G.ic[1] - 1 + 31) / 32, (G.ic[0] - 1 + 7) / 8);
            launch_dependent(fits(g) ? k_adv_mass2<false> : k_adv_mass2<true>, grid_of(g), 256, 0, st, G, g, F, fl[0].f[4], fl[1].f[4]);
        }
    }
    // advect (explicit.py:5-74): every axis is swept twice; the face arrays keep the fluxes of the
    // second sweep, so the first does not write them
    void strang(double dt, int odd) {
        const int nd = G.nd;
        for (int q = 0; q < 2 * nd; ++q) {
            const int up = q < nd ? q : 2 * nd - 1 - q;
            const int s = odd ? up : nd - 1 - up;
            sweep<false>(s, 0.5 * dt / G.d[s], q >= nd);
        }
        for (int s = 0; s < nd; ++s) bd(s);
    }
    // advect_rk (explicit.py:160-257): fluxes of all axes from the start state, then the updates.
    // The boundary data after each flux (explicit.py:155) would rewrite the same values.
    void rk(double dt) {
        const int nd = G.nd;
        for (int s = 0; s < nd; ++s) sweep<true>(s, 0.0, 1);
        const double lx = dt / G.d[0], ly = dt / G.d[1], lz = dt / G.d[2];
        const dim3 blk(32, 8);
        const TileRow g = nd == 3 ? tile_row((G.ic[2] + 31) / 32, (G.ic[1] + 7) / 8, (G.ic[0] + UPD_X - 1) / UPD_X)
                                  : tile_row((G.ic[1] + 31) / 32, (G.ic[0] + 7) / 8);
        const auto k = fits(g) ? (nd == 3 ? k_adv_update<3, false> : k_adv_update<2, false>)
                               : (nd == 3 ? k_adv_update<3, true> : k_adv_update<2, true>);
        launch_dependent(k, grid_of(g), blk, 0, st, G, g, F, fl[0], fl[1], fl[2], lx, ly, lz, pw);
        for (int s = 0; s < nd; ++s) bd(s);
    }
};

bool adv_setup(const bella_adv2d *a, DevEx &ex, void *stream) {
    if (!a || a->inx < 5 || a->iny < 5) return false;
    const double *req[] = {a->rho, a->rhou, a->rhov, a->rhow, a->rhoY, a->rhoX, a->hydro_rhoY0, a->strat_inv};
    for (const double *p : req)
        if (!p) return false;
    for (int q = 0; q < 6; ++q)
        if (!a->fx[q] || !a->fy[q]) return false;
    AdvGeom &G = ex.G;
    G.nd = 2;
    G.ic[0] = a->inx + 3; G.ic[1] = a->iny + 3; G.ic[2] = 1;
    G.bc[0] = a->x_wall ? 1 : 0; G.bc[1] = a->y_wall ? 1 : 0; G.bc[2] = 0;
    G.d[0] = a->dx; G.d[1] = a->dy; G.d[2] = 1.0;
    G.g = a->g; G.gamm = a->gamm; G.is_compressible = a->is_compressible;
    double *f[6] = {a->rho, a->rhou, a->rhov, a->rhow, a->rhoY, a->rhoX};
    for (int q = 0; q < 6; ++q) {
        ex.F.f[q] = f[q];
        ex.fl[0].f[q] = a->fx[q];
        ex.fl[1].f[q] = a->fy[q];
        ex.fl[2].f[q] = nullptr;
    }
    ex.rhoY0 = a->hydro_rhoY0; ex.strat_inv = a->strat_inv; ex.pw = a->pwchi;
    ex.st = (cudaStream_t)stream;
    return true;
}

bool adv_setup(const bella_adv3d *a, DevEx &ex, void *stream) {
    if (!a || a->inx < 5 || a->iny < 5 || a->inz < 5) return false;
    const double *req[] = {a->rho, a->rhou, a->rhov, a->rhow, a->rhoY, a->rhoX, a->hydro_rhoY0, a->strat_inv};
    for (const double *p : req)
        if (!p) return false;
    for (int q = 0; q < 6; ++q)
        if (!a->fx[q] || !a->fy[q] || !a->fz[q]) return false;
    AdvGeom &G = ex.G;
    G.nd = 3;
    G.ic[0] = a->inx + 3; G.ic[1] = a->iny + 3; G.ic[2] = a->inz + 3;
    G.bc[0] = a->x_wall ? 1 : 0; G.bc[1] = a->y_wall ? 1 : 0; G.bc[2] = a->z_wall ? 1 : 0;
    G.d[0] = a->dx; G.d[1] = a->dy; G.d[2] = a->dz;
    G.g = a->g; G.gamm = a->gamm; G.is_compressible = a->is_compressible;
    double *f[6] = {a->rho, a->rhou, a->rhov, a->rhow, a->rhoY, a->rhoX};
    for (int q = 0; q < 6; ++q) {
        ex.F.f[q] = f[q];
        ex.fl[0].f[q] = a->fx[q];
        ex.fl[1].f[q] = a->fy[q];
        ex.fl[2].f[q] = a->fz[q];
    }
    ex.rhoY0 = a->hydro_rhoY0; ex.strat_inv = a->strat_inv; ex.pw = a->pwchi;
    ex.st = (cudaStream_t)stream;
    return true;
}

}  // namespace
}  // namespace bella

using namespace bella;

template <class A>
static int fluxes_impl(const A *a, void *stream) {
    DevEx ex;
    if (!adv_setup(a, ex, stream)) return BELLA_EINVAL;
    ex.mass();
    return cudaGetLastError() == cudaSuccess ? BELLA_OK : BELLA_ECUDA;
}

template <class A>
static int advect_impl(const A *a, double dt, int odd, void *stream) {
    DevEx ex;
    if (!adv_setup(a, ex, stream)) return BELLA_EINVAL;
    ex.strang(dt, odd);
    return cudaGetLastError() == cudaSuccess ? BELLA_OK : BELLA_ECUDA;
}

template <class A>
static int advect_rk_impl(const A *a, double dt, void *stream) {
    DevEx ex;
    if (!adv_setup(a, ex, stream)) return BELLA_EINVAL;
    ex.rk(dt);
    return cudaGetLastError() == cudaSuccess ? BELLA_OK : BELLA_ECUDA;
}

// set_explicit_boundary_data (boundary.py:7-216) of the whole state: axis by axis
template <class A>
static int boundary_impl(const A *a, void *stream) {
    DevEx ex;
    if (!adv_setup(a, ex, stream)) return BELLA_EINVAL;
    for (int s = 0; s < ex.G.nd; ++s) ex.bd(s);
    return cudaGetLastError() == cudaSuccess ? BELLA_OK : BELLA_ECUDA;
}

extern "C" {
int bella_advective_fluxes2d(const bella_adv2d *a, void *stream) { return fluxes_impl(a, stream); }
int bella_advect2d(const bella_adv2d *a, double dt, int odd, void *stream) { return advect_impl(a, dt, odd, stream); }
int bella_advect_rk2d(const bella_adv2d *a, double dt, void *stream) { return advect_rk_impl(a, dt, stream); }
int bella_boundary2d(const bella_adv2d *a, void *stream) { return boundary_impl(a, stream); }
int bella_advective_fluxes3d(const bella_adv3d *a, void *stream) { return fluxes_impl(a, stream); }
int bella_advect3d(const bella_adv3d *a, double dt, int odd, void *stream) { return advect_impl(a, dt, odd, stream); }
int bella_advect_rk3d(const bella_adv3d *a, double dt, void *stream) { return advect_rk_impl(a, dt, stream); }
int bella_boundary3d(const bella_adv3d *a, void *stream) { return boundary_impl(a, stream); }
}
