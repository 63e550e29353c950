// bella_proj3d.cu -- the 3D implicit nodal projection on the device.
//
// The reference's projection pieces are dimension-generic and run in 3D; its
// step (second_projection.py:97-277) cannot (the 3D branch uses diag_inv and p2
// before assignment, :183-203).  bella_projection3d assembles the step from the
// 3D pieces with the glue of the reference's 2D branch: unknowns are the inner
// nodes, hplus the cells around them, hcenter and diag_inv (the 3D
// precon_diag_prepare) at those nodes, the right-hand side the node.isc
// divergence scaled by 1/dt and diag_inv, vector order C over (x, y, z)
// (second_projection.py:224), corrf = dt * coriolis_strength[0] (laplacian.py:894).
//
// Kernels (what bounds them: bella_cells3d.cuh):
//   adv_boundary      set_explicit_boundary_data (bella_advect.cu)   boundary.py:7-281
//   k3_coeff          wplus (all three axes) -> packed cell plane    second_projection.py:308-341
//                     wcenter, wall scaling, regime, 3D diagonal     :343-356, :147-153, laplacian.py:1284-1356
//   k3_zero_ghost     y-wall ghost momenta of divergence_nodes       :542-551
//   k3_divergence     divergence_nodes (3D branch), /dt, *diag_inv   :556-570, :139, :170
//   k3_ghost          set_ghostnodes_p2 along one axis               boundary.py:296-369
//   k3_correction     grad_nodes + correction_nodes (3D)             :280-306, :496-521, :604-646
//   k3_scatter, k3_add   p2_full[i2] = x; p2_nodes += p2_full        :265-275
// Array layout: the reference's NumPy C order over (x, y, z), ghosts included.
#include <cstring>

#include "bella_advect.cuh"
#include "bella_cells3d.cuh"

namespace bella {

struct Proj3Dev {
    int icx, icy, icz;     // cells incl. ghosts (inx+3, iny+3, inz+3)
    int ncx, ncy, ncz;     // nodes incl. ghosts (inx+4, iny+4, inz+4)
    int bc[3];             // 0 periodic, 1 wall
    double dx, dy, dz, dt, Msq, g, gamm, compressibility;
    double Ginv, cexp;     // gamma / (gamma - 1), 2 - gamma
    double ccenter, wdiag; // wcenter's factor on the sum of eight cells; the diagonal's on wplus's sum
    double cx, cy, cz;     // 0.25 / spacing; cx with the sign of the divergence's x term: -1 as
                           // divergence_nodes' 3D branch, +1 as its 2D branch
    Coriolis3 cor;
    int is_compressible;
};

__device__ __forceinline__ long long c3(const Proj3Dev &P, int i, int j, int k) {
    return ((long long)i * P.icy + j) * P.icz + k;
}
__device__ __forceinline__ long long n3(const Proj3Dev &P, int i, int j, int k) {
    return ((long long)i * P.ncy + j) * P.ncz + k;
}

// dS/dy on cell plane j from the node background S0 (variable.py:162-177)
__device__ __forceinline__ double dSdy3(const Proj3Dev &P, const double *S0n, int j) {
    return (S0n[j + 1] - S0n[j]) / P.dy;
}

// Coefficients of the operator in one pass over the coefficient state.  Cells: wplus =
// Gammainv * rhoY * Y, those around the inner nodes packed (inx+1)(iny+1)(inz+1) for the operator
// (the same plane serves hplusx, hplusy, hplusz).  Nodes (node.isc): wcenter = ccenter *
// box(rhoY^(2-gamma)) / 8, halved on wall rows, times compressibility in the pseudo-incompressible
// regime; the 3D Jacobi diagonal (laplacian.py:1334-1356: coefficient 0.0625, the x-y
// cross terms kept as the reference has them); inner nodes packed -> hc, dinv.
// A block walks an 8x32 tile of nodes along x, the cells of a plane in shared memory: 0.62 ms at
// 257x129x257 nodes, against 1.79 (a pow per cell) + 1.35 ms (sixteen reads and seven
// divisions a node) as two passes.
__global__ void __launch_bounds__(C3_THREADS)
k3_coeff(Proj3Dev P, Walk3 walk, const double *rhoC, const double *rhoYC, double *hpk, double *dinv_isc, double *hc,
         double *dinv) {
    constexpr int NJ = C3_J + 1, NK = C3_K + 1, NE = NJ * NK;
    __shared__ double sm[2][2][NE];
    const int nix = P.icx - 1, niy = P.icy - 1, niz = P.icz - 1;
    const int t = threadIdx.x, tk = t % C3_K, tj = t / C3_K;
    const uint3 tile = tile_of(walk.tiles);
    const int k0 = tile.x * C3_K, j0 = tile.y * C3_J;
    const int a0 = tile.z * walk.seg, a1 = a0 + walk.seg < nix ? a0 + walk.seg : nix;
    const int b = j0 + tj, c = k0 + tk;
    const bool on = b < niy && c < niz;
    const double weight = P.is_compressible == 1 ? 1.0 : P.compressibility;   // second_projection.py:147-153
    double w1 = 0.0, q1 = 0.0;
    int buf = 0;
    for (int p = a0; p <= a1; ++p, buf ^= 1) {
        for (int e = t; e < NE; e += C3_THREADS) {
            const int lj = e / NK, lk = e - lj * NK, j = j0 + lj, k = k0 + lk;
            if (j < P.icy && k < P.icz) {
                const long long x = c3(P, p, j, k);
                const double rY = rhoYC[x], w = P.Ginv * rY * (rY / rhoC[x]);
                sm[buf][0][e] = w;
                sm[buf][1][e] = weighted_pow(rY, P.cexp, weight);
                // each cell belongs to the tile that holds it as a lower corner
                if (lj < C3_J && lk < C3_K && p < (a1 == nix ? P.icx : a1) && p >= 1 && p <= P.icx - 2 && j >= 1 &&
                    j <= P.icy - 2 && k >= 1 && k <= P.icz - 2)
                    hpk[((long long)(p - 1) * (P.icy - 2) + (j - 1)) * (P.icz - 2) + (k - 1)] = w;
            }
        }
        __syncthreads();                                // the other buffer's readers are past it
        const int e = tj * NK + tk;
        const double *sw = sm[buf][0], *sq = sm[buf][1];
        const double w = (sw[e] + sw[e + 1]) + (sw[e + NK] + sw[e + NK + 1]);
        const double q = (sq[e] + sq[e + 1]) + (sq[e + NK] + sq[e + NK + 1]);
        if (on && p > a0) {
            const int a = p - 1;
            const double wc = P.ccenter * (q1 + q) * node_wall_scale(P, a, b, c, 0.5) * weight;
            const double di = 1.0 / (wc - P.wdiag * (w1 + w));
            dinv_isc[((long long)a * niy + b) * niz + c] = di;
            if (a >= 1 && a <= nix - 2 && b >= 1 && b <= niy - 2 && c >= 1 && c <= niz - 2) {
                const long long pk = ((long long)(a - 1) * (niy - 2) + (b - 1)) * (niz - 2) + (c - 1);
                hc[pk] = wc;
                dinv[pk] = di;
            }
        }
        w1 = w; q1 = q;
    }
}

// divergence_nodes at a y wall: momenta of the two ghost planes on each side zeroed
__global__ void k3_zero_ghost(Proj3Dev P, double *rhou, double *rhov, double *rhow) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)P.icx * P.icz || P.bc[1] != 1) return;
    const int i = (int)(e / P.icz), k = (int)(e - (long long)i * P.icz);
    const int n = P.icy;
    const int rows[4] = {0, 1, n - 2, n - 1};
    for (int t = 0; t < 4; ++t) {
        const long long q = c3(P, i, rows[t], k);
        rhou[q] = 0.0;
        rhov[q] = 0.0;
        rhow[q] = 0.0;
    }
}

// divergence_nodes, 3D branch (second_projection.py:556-570) on node.isc, with the
// reference's sign on the x term (Ux = -0.5 * (...), :563) or the 2D branch's
// (in cx); /dt (:139), b = (rhs * diag_inv)[inner] in C order (:170, :224).  The regime mix
// (:149-150) adds up to the same right-hand side.  0.61 ms at 257x129x257 nodes, against 2.46
// ms with 24 products and twelve divisions a node.
__global__ void __launch_bounds__(C3_THREADS)
k3_divergence(Proj3Dev P, Walk3 walk, const double *rho, const double *rhou, const double *rhov, const double *rhow,
              const double *rhoY, const double *dinv_isc, double *rhs_isc, double *bvec) {
    const int nix = P.icx - 1, niy = P.icy - 1, niz = P.icz - 1;
    const double s = 1.0 / P.dt;
    walk_divergence<false>(P, walk, rho, rhou, rhov, rhow, rhoY, s * P.cx, s * P.cy, s * P.cz, 0.0, 0.0,
        [&](int a, int b, int c, double rhs, double) {
            const long long e = ((long long)a * niy + b) * niz + c;
            rhs_isc[e] = rhs;
            if (a >= 1 && a <= nix - 2 && b >= 1 && b <= niy - 2 && c >= 1 && c <= niz - 2)
                bvec[((long long)(a - 1) * (niy - 2) + (b - 1)) * (niz - 2) + (c - 1)] = rhs * dinv_isc[e];
        });
}

// set_ghostnodes_p2 along axis dim: periodic_plus_one (boundary.py:348-369) or
// 'reflect', one thread per line of nodes along dim
__global__ void k3_ghost(Proj3Dev P, int dim, double *p) {
    const int ext[3] = {P.ncx, P.ncy, P.ncz};
    const int da = dim == 0 ? 1 : 0, db = dim == 2 ? 1 : 2;
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)ext[da] * ext[db]) return;
    int c[3];
    c[da] = (int)(e / ext[db]);
    c[db] = (int)(e - (long long)c[da] * ext[db]);
    const int n = ext[dim];
    auto at = [&](int t) -> double & {
        c[dim] = t;
        return p[n3(P, c[0], c[1], c[2])];
    };
    if (P.bc[dim] == 0) {
        const double h0 = at(n - 5), h1 = at(n - 4), h2 = at(n - 3);
        const double t0 = at(2), t1 = at(3), t2 = at(4);
        at(0) = h0; at(1) = h1; at(2) = h2;
        at(n - 3) = t0; at(n - 2) = t1; at(n - 1) = t2;
    } else {
        at(0) = at(4);
        at(1) = at(3);
        at(n - 2) = at(n - 4);
        at(n - 1) = at(n - 5);
    }
}

// correction_nodes (second_projection.py:280-306) with the 3D grad_nodes (:496-521)
// and the Coriolis inverse (:604-646), on every cell.  A thread walks its (y, z) row
// along x and keeps the last node plane's sums.  With Y = rhoY / rho the factor
// (rho / rhoY) * Gammainv * rhoY * Y of the gradient is Gammainv * rhoY, so without Coriolis forces
// a cell needs one division; where rho or rhoY is zero or not finite nothing cancels, and the formula
// stands as it is.  0.72 ms at 257x129x257 nodes, against 2.25
// ms with eight node reads and nine divisions a cell.
__global__ void __launch_bounds__(C3_THREADS)
k3_correction(Proj3Dev P, Walk3 walk, const double *p, const double *rho, double *rhou, double *rhov, double *rhow,
              const double *rhoY, double *rhoX, const double *S0n, double updt_chi) {
    const uint3 tile = tile_of(walk.tiles);
    const int k = tile.x * C3_K + threadIdx.x % C3_K, j = tile.y * C3_J + threadIdx.x / C3_K;
    if (j >= P.icy || k >= P.icz) return;
    const int i0 = tile.z * walk.seg, i1 = i0 + walk.seg < P.icx ? i0 + walk.seg : P.icx;
    const double ds = dSdy3(P, S0n, j);
    const double ux = -P.dt * P.Ginv * 0.25 / P.dx, uy = -P.dt * P.Ginv * 0.25 / P.dy, uz = -P.dt * P.Ginv * 0.25 / P.dz;
    const double nu_y = -P.dt * P.dt * (P.g / P.Msq) * ds;      // nu = nu_y * rhoY / rho
    const double chi = -updt_chi * P.dt * ds;
    PlaneGrad a = plane_grad(p, n3(P, i0, j, k), P.ncz);
    for (int i = i0; i < i1; ++i) {
        const long long e = c3(P, i, j, k);
        const double rY = rhoY[e], r = rho[e];
        const PlaneGrad b = plane_grad(p, n3(P, i + 1, j, k), P.ncz);
        double U = ux * rY * (b.x - a.x), V = uy * rY * (a.y + b.y), W = uz * rY * (a.z + b.z);
        const double qr = P.cor.nh * r + nu_y * rY;             // (nu + nonhydro) rho
        if (!is_normal(r) || !is_normal(rY)) {                  // nothing cancels
            const double Y = rY / r, thinv = r / rY;
            U *= Y; V *= Y; W *= Y;
            cor_apply(P.cor, nu_y * Y + P.cor.nh, U, V, W);
            U *= thinv; V *= thinv; W *= thinv;
        } else if (cor_diagonal(P.cor, qr, U, V, W)) {
            V = P.cor.nh * V * r / qr;
        } else {
            cor_apply(P.cor, qr / r, U, V, W);
        }
        rhou[e] += U;
        const double rv = rhov[e] + V;
        rhov[e] = rv;
        rhow[e] += W;
        rhoX[e] += chi * rv;
        a = b;
    }
}

// p2_full = 0; p2_full[2:-2, 2:-2, 2:-2] = x.reshape(inx, iny, inz)
__global__ void k3_scatter(Proj3Dev P, const double *x, double *pfull) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)P.ncx * P.ncy * P.ncz) return;
    const int i = (int)(e / ((long long)P.ncy * P.ncz));
    const int r = (int)(e - (long long)i * P.ncy * P.ncz);
    const int j = r / P.ncz, k = r - j * P.ncz;
    const int inx = P.ncx - 4, iny = P.ncy - 4, inz = P.ncz - 4;
    double v = 0.0;
    if (i >= 2 && i < 2 + inx && j >= 2 && j < 2 + iny && k >= 2 && k < 2 + inz)
        v = x[((long long)(i - 2) * iny + (j - 2)) * inz + (k - 2)];
    pfull[e] = v;
}

__global__ void k3_add(long long n, double *a, const double *b) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e < n) a[e] += b[e];
}

}  // namespace bella

using namespace bella;

static int grid3(long long n) { return (int)((n + 255) / 256); }

static void bd3(const Proj3Dev &P, double *const F[6], const double *rhoY0, const double *strat_inv,
                cudaStream_t s, long long &launches) {
    AdvGeom G;
    G.nd = 3;
    G.ic[0] = P.icx; G.ic[1] = P.icy; G.ic[2] = P.icz;
    for (int d = 0; d < 3; ++d) G.bc[d] = P.bc[d];
    G.d[0] = P.dx; G.d[1] = P.dy; G.d[2] = P.dz;
    G.g = P.g; G.gamm = P.gamm; G.is_compressible = P.is_compressible;
    AdvFields A;
    for (int q = 0; q < 6; ++q) A.f[q] = F[q];
    for (int d = 0; d < 3; ++d) adv_boundary(G, d, A, rhoY0, strat_inv, s);
    launches += 3;
}

static void ghost3(const Proj3Dev &P, double *p, cudaStream_t s, long long &launches) {
    k3_ghost<<<grid3((long long)P.ncy * P.ncz), 256, 0, s>>>(P, 0, p);
    k3_ghost<<<grid3((long long)P.ncx * P.ncz), 256, 0, s>>>(P, 1, p);
    k3_ghost<<<grid3((long long)P.ncx * P.ncy), 256, 0, s>>>(P, 2, p);
    launches += 3;
}

extern "C" int bella_projection3d(bella_ws *ws, const bella_proj3d *a, const bella_solve_opts *opts,
                                  bella_solve_stats *stats, void *stream) {
    if (!ws || !a) return BELLA_EINVAL;
    if (a->inx < 5 || a->iny < 5 || a->inz < 5 || !a->rho || !a->rhou || !a->rhov || !a->rhow || !a->rhoY ||
        !a->rhoX || !a->p2 || !a->hydro_rhoY0 || !a->S0n || !a->strat_inv)
        return BELLA_EINVAL;
    if (a->precond != 0 && (a->precond != 1 || !a->y_wall)) return BELLA_EINVAL;
    cudaStream_t s = (cudaStream_t)stream;
    Proj3Dev P;
    P.icx = a->inx + 3; P.icy = a->iny + 3; P.icz = a->inz + 3;
    P.ncx = a->inx + 4; P.ncy = a->iny + 4; P.ncz = a->inz + 4;
    P.bc[0] = a->x_wall ? 1 : 0; P.bc[1] = a->y_wall ? 1 : 0; P.bc[2] = a->z_wall ? 1 : 0;
    P.dx = a->dx; P.dy = a->dy; P.dz = a->dz; P.dt = a->dt; P.Msq = a->Msq; P.g = a->g; P.gamm = a->gamm;
    P.compressibility = a->compressibility;
    P.is_compressible = a->is_compressible;
    P.Ginv = a->gamm / (a->gamm - 1.0);
    P.cexp = 2.0 - a->gamm;
    P.ccenter = -a->Msq / (a->gamm - 1.0) / (a->dt * a->dt) / 8.0;
    const double cf = 0.0625;
    P.wdiag = cf / (a->dx * a->dx) + cf / (a->dy * a->dy) + 2.0 * (cf / (a->dx * a->dy)) + cf / (a->dz * a->dz);
    P.cx = (a->div_sign_2d ? 0.25 : -0.25) / a->dx; P.cy = 0.25 / a->dy; P.cz = 0.25 / a->dz;
    P.cor = coriolis3(a->dt, a->nonhydro, a->coriolis);
    const long long nnode = (long long)P.ncx * P.ncy * P.ncz;
    const long long nisc = (long long)(P.icx - 1) * (P.icy - 1) * (P.icz - 1);
    const long long nin = (long long)a->inx * a->iny * a->inz;
    const long long npk = (long long)(a->inx + 1) * (a->iny + 1) * (a->inz + 1);
    // scratch: dinv_isc, rhs_isc, packed cells, hc, dinv, b, x, pfull
    const size_t need = (size_t)(2 * nisc + npk + 4 * nin + nnode);
    if (ws->proj_cap < need) {
        cudaFree(ws->proj_buf);
        ws->proj_buf = nullptr;
        ws->proj_cap = 0;
        if (cudaMalloc(&ws->proj_buf, need * sizeof(double)) != cudaSuccess) return BELLA_ECUDA;
        ws->proj_cap = need;
    }
    double *q = ws->proj_buf;
    double *dinv_isc = q; q += nisc;
    double *rhs_isc = q; q += nisc;
    double *hpk = q; q += npk;
    double *hc = q; q += nin;
    double *dinv = q; q += nin;
    double *bvec = q; q += nin;
    double *xvec = q; q += nin;
    double *pfull = q;

    const bool has0 = a->rho0 != nullptr;
    double *const F[6] = {a->rho, a->rhou, a->rhov, a->rhow, a->rhoY, a->rhoX};
    double *const C[6] = {has0 ? a->rho0 : a->rho, has0 ? a->rhou0 : a->rhou, has0 ? a->rhov0 : a->rhov,
                          has0 ? a->rhow0 : a->rhow, has0 ? a->rhoY0 : a->rhoY, has0 ? a->rhoX0 : a->rhoX};
    long long L = 0;
    // 1. coefficient state: boundary data of Sol0 or Sol (second_projection.py:113-118)
    bd3(P, C, a->hydro_rhoY0, a->strat_inv, s, L);
    // 2. ghost nodes of p2, correction with the old p2, boundary data (:130-132)
    ghost3(P, a->p2, s, L);
    const Walk3 cells = walk3(P.icx, P.icy, P.icz, 1), nodes = walk3(P.icx - 1, P.icy - 1, P.icz - 1, 1);
    k3_correction<<<cells.tiles.blocks, C3_THREADS, 0, s>>>(P, cells, a->p2, a->rho, a->rhou, a->rhov, a->rhow, a->rhoY,
                                                    a->rhoX, a->S0n, 0.0);
    bd3(P, F, a->hydro_rhoY0, a->strat_inv, s, L);
    // 3. coefficients from the coefficient state and the diagonal
    k3_coeff<<<nodes.tiles.blocks, C3_THREADS, 0, s>>>(P, nodes, C[0], C[4], hpk, dinv_isc, hc, dinv);
    // 4. divergence right-hand side (:134-170, :224)
    k3_zero_ghost<<<grid3((long long)P.icx * P.icz), 256, 0, s>>>(P, a->rhou, a->rhov, a->rhow);
    k3_divergence<<<nodes.tiles.blocks, C3_THREADS, 0, s>>>(P, nodes, a->rho, a->rhou, a->rhov, a->rhow, a->rhoY, dinv_isc,
                                                    rhs_isc, bvec);
    L += 4;
    if (a->rhs_out) cudaMemcpyAsync(a->rhs_out, rhs_isc, nisc * sizeof(double), cudaMemcpyDeviceToDevice, s);
    ws->launches += L;
    if (cudaGetLastError() != cudaSuccess) return BELLA_ECUDA;
    // 5. operator (the closure of stencil_27pt, laplacian.py:872-896) and solve (:230)
    const bool hc_on = !(a->is_compressible == 0 && a->compressibility == 0.0);
    bella_op3d op;
    op.nx = a->inx; op.ny = a->iny; op.nz = a->inz;
    op.x_wall = a->x_wall; op.y_wall = a->y_wall; op.z_wall = a->z_wall;
    op.dx = a->dx; op.dy = a->dy; op.dz = a->dz;
    op.corrf = a->dt * a->coriolis[0];
    op.hplusx = hpk; op.hplusy = hpk; op.hplusz = hpk;
    op.hcenter = hc_on ? hc : nullptr;
    op.diag_inv = dinv;
    int rc = bella_op3d_set(ws, &op, stream);
    if (rc != BELLA_OK) return rc;
    bella_solve_opts o;
    if (opts) o = *opts; else bella_solve_opts_default(&o);
    o.x0_zero = 1;
    int st;
    if (a->precond == 1) {
        // the workspace's background solve, re-derived from this call's coefficients
        // (made anew when the grid or a boundary kind changed)
        if (!ws->sp_cache || bella_spectral3d_update(ws->sp_cache, &op, stream) != BELLA_OK) {
            bella_spectral3d_destroy(ws->sp_cache);
            ws->sp_cache = nullptr;
            rc = bella_spectral3d_create(&ws->sp_cache, &op, ws->device, stream);
            if (rc != BELLA_OK) return rc;
        }
        st = bella_fbicgstab_pc(ws, ws->sp_cache, nullptr, 0, bvec, xvec, &o, stats, stream);
    } else {
        st = bella_bicgstab(ws, bvec, xvec, &o, stats, stream);
    }
    if (st < 0) return st;
    // 6. p2_full, ghost nodes, correction with updt_chi = 1, p2 += p2_full, ghosts, boundary data (:265-277)
    L = 0;
    k3_scatter<<<grid3(nnode), 256, 0, s>>>(P, xvec, pfull);
    ghost3(P, pfull, s, L);
    k3_correction<<<cells.tiles.blocks, C3_THREADS, 0, s>>>(P, cells, pfull, a->rho, a->rhou, a->rhov, a->rhow, a->rhoY,
                                                    a->rhoX, a->S0n, 1.0);
    k3_add<<<grid3(nnode), 256, 0, s>>>(nnode, a->p2, pfull);
    ghost3(P, a->p2, s, L);
    bd3(P, F, a->hydro_rhoY0, a->strat_inv, s, L);
    ws->launches += L + 3;
    if (cudaGetLastError() != cudaSuccess) return BELLA_ECUDA;
    return st;
}
