// bella_expl3d.cu -- the explicit parts of the 3D projection on the device:
// euler_forward_non_advective (second_projection.py:22-74, with the 2D branch's
// glue: the divergence on node.isc) and euler_backward_non_advective_expl_part
// (:77-92).  The arithmetic is bella_expl3d.cuh's (checked on the CPU by
// tests/test_expl3d_host.py); boundary data (:72, :92) are the advection's (adv_boundary),
// which restate set_explicit_boundary_data axis by axis.
//   k_e3_zero_ghost   divergence_nodes' y-wall ghost momenta            :542-551
//   k_e3_fw_nodes     divergence, wall doubling, pressure increment     :39-47, :66
//   k_e3_fw_cells     momenta and rhoX from the old p2                   :49-64
//   k_e3_fw_p2        p2 += compressibility * increment                  :68-69
//   k_e3_ghost        ghost nodes of p2 along one axis                   :71
//   k_e3_xp_cells     buoyancy, wind, Coriolis inverse                   :82-90
#include "bella_advect.cuh"
#include "bella_expl3d.cuh"
#include "bella_cells3d.cuh"

namespace bella {

__global__ void k_e3_zero_ghost(Expl3Geom G, Expl3Fields F) {
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)G.icx * G.icz || G.bc[1] != 1) return;
    const int i = (int)(e / G.icz), k = (int)(e - (long long)i * G.icz);
    const int rows[4] = {0, 1, G.icy - 2, G.icy - 1};
    for (int t = 0; t < 4; ++t) {
        const long long c = e3_cell(G, i, rows[t], k);
        F.f[1][c] = 0.0;
        F.f[2][c] = 0.0;
        F.f[3][c] = 0.0;
    }
}

// divergence of the momenta with the wall rows doubled (:39-40) and the pressure increment
// dp = -dt * dpidP * div (:45-47, :66), as e3_forward_node.  0.74 ms at 257x129x257
// nodes, against 15.1 ms with eight pow and 36 divisions a node.
__global__ void __launch_bounds__(C3_THREADS)
k_e3_fw_nodes(Expl3Geom G, Walk3 walk, double cx, double cy, double cz, double kdp, Expl3Fields F, double *rhs, double *dp) {
    const int ny = G.icy - 1, nz = G.icz - 1;
    walk_divergence<true>(G, walk, F.f[0], F.f[1], F.f[2], F.f[3], F.f[4], cx, cy, cz, G.gamm - 2.0, G.compressibility,
        [&](int a, int b, int c, double div, double s) {
            const long long e = ((long long)a * ny + b) * nz + c;
            div *= node_wall_scale(G, a, b, c, 2.0);
            if (rhs) rhs[e] = div;
            dp[e] = kdp * s * div;
        });
}

// momenta from the pressure gradient of the old p2, buoyancy and Coriolis of the
// background-wind deviations, rhoX from the background (:49-64), as e3_forward_cell: a
// thread walks its (y, z) row along x.  1.0 ms at 257x129x257 nodes, against 2.0 ms
// with nine divisions a cell.
__global__ void __launch_bounds__(C3_THREADS)
k_e3_fw_cells(Expl3Geom G, Walk3 walk, Expl3Fields F, const double *p2, const double *S0c, const double *S0n) {
    const uint3 tile = tile_of(walk.tiles);
    const int k = tile.x * C3_K + threadIdx.x % C3_K, j = tile.y * C3_J + threadIdx.x / C3_K;
    if (j >= G.icy || k >= G.icz) return;
    const int i0 = tile.z * walk.seg, i1 = i0 + walk.seg < G.icx ? i0 + walk.seg : G.icx;
    const double Ginv = G.gamm / (G.gamm - 1.0);
    const double gx = Ginv * 0.25 / G.dx, gy = Ginv * 0.25 / G.dy, gz = Ginv * 0.25 / G.dz;
    const double dSdy = (S0n[j + 1] - S0n[j]) / G.dy, buoy = G.g / G.Msq * G.nonhydro, ak = 1 - G.is_ArakawaKonor;
    const double ch1 = G.cor[0], cv = G.cor[1], ch2 = G.cor[2];
    PlaneGrad a = plane_grad(p2, e3_node(G, i0, j, k), G.icz + 1);
    for (int i = i0; i < i1; ++i) {
        const long long e = e3_cell(G, i, j, k);
        const double rho = F.f[0][e], ru = F.f[1][e], rv = F.f[2][e], rw = F.f[3][e], rY = F.f[4][e], rX = F.f[5][e];
        const PlaneGrad b = plane_grad(p2, e3_node(G, i + 1, j, k), G.icz + 1);
        const double Y = rY / rho;
        const double drhou = ru - G.wind[0] * rho, drhov = rv - G.wind[1] * rho, drhow = rw - G.wind[2] * rho;
        F.f[1][e] = ru - G.dt * (gx * rY * (b.x - a.x) - ch2 * drhov + cv * drhow);
        F.f[2][e] = rv - G.dt * (gy * rY * (a.y + b.y) + buoy * (Y * rX) - ch1 * drhow + ch2 * drhou) * ak;
        F.f[3][e] = rw - G.dt * (gz * rY * (a.z + b.z) - cv * drhou + ch1 * drhov);
        const double vr = is_normal(rho) ? rv : rv / rho * rho;          // v rho
        F.f[5][e] = rho * (rho / rY - S0c[e]) - G.dt * dSdy * vr;
        a = b;
    }
}

__global__ void k_e3_fw_p2(Expl3Geom G, const double *dp, double *p2) {
    const int nx = G.icx - 1, ny = G.icy - 1, nz = G.icz - 1;
    const long long e = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (e >= (long long)nx * ny * nz) return;
    const int a = (int)(e / ((long long)ny * nz));
    const int r = (int)(e - (long long)a * ny * nz);
    const int b = r / nz, c = r - b * nz;
    const long long n = e3_node(G, a + 1, b + 1, c + 1);
    p2[n] += G.compressibility * dp[e];
}

__global__ void k_e3_ghost(Expl3Geom G, int d, double *p) {
    const int nn[3] = {G.icx + 1, G.icy + 1, G.icz + 1};
    const long long nl = (long long)nn[d == 0 ? 1 : 0] * nn[d == 2 ? 1 : 2];
    const long long l = blockIdx.x * (long long)blockDim.x + threadIdx.x;
    if (l < nl) e3_ghost_line(G, d, l, p);
}

// buoyancy into rhov, background wind off, the implicit Coriolis / buoyancy inverse, background wind
// on (:77-92), as e3_expl_part_cell.  Without Coriolis forces and wind the inverse leaves rhou and rhow as
// they are (cor_diagonal), and so does this kernel, with one division a cell: 0.30 ms at 257x129x257 nodes, against 1.36 ms
// with seven divisions a cell.
__global__ void __launch_bounds__(C3_THREADS)
k_e3_xp_cells(Expl3Geom G, Walk3 walk, Coriolis3 cor, Expl3Fields F, const double *S0n) {
    const uint3 tile = tile_of(walk.tiles);
    const int k = tile.x * C3_K + threadIdx.x % C3_K, j = tile.y * C3_J + threadIdx.x / C3_K;
    if (j >= G.icy || k >= G.icz) return;
    const int i0 = tile.z * walk.seg, i1 = i0 + walk.seg < G.icx ? i0 + walk.seg : G.icx;
    const double strat = (S0n[j + 1] - S0n[j]) / G.dy, gM = G.g / G.Msq;
    const double nu_y = -(G.dt * G.dt) * gM * strat, kb = G.dt * gM;
    const bool wind = G.wind[0] != 0.0 || G.wind[1] != 0.0 || G.wind[2] != 0.0;
    for (int i = i0; i < i1; ++i) {
        const long long e = e3_cell(G, i, j, k);
        const double rho = F.f[0][e], rY = F.f[4][e];
        const double ru = F.f[1][e], rv = F.f[2][e], rw = F.f[3][e], rX = F.f[5][e];
        const double qr = cor.nh * rho + nu_y * rY;             // (nu + nonhydro) rho
        const double vr = cor.nh * rv * rho - kb * (rY * rX);   // v rho
        const bool usual = is_normal(rho) && is_normal(rY);
        if (!wind && usual && cor_diagonal(cor, qr, ru, vr, rw)) {
            F.f[2][e] = cor.nh * vr / qr;
            continue;
        }
        double V = cor.nh * rv - kb * (rY * (rX / rho));
        double U = ru - G.wind[0] * rho, W = rw - G.wind[2] * rho;
        V -= G.wind[1] * rho;
        cor_apply(cor, usual ? qr / rho : nu_y * (rY / rho) + cor.nh, U, V, W);
        F.f[1][e] = U + G.wind[0] * rho;
        F.f[2][e] = V + G.wind[1] * rho;
        F.f[3][e] = W + G.wind[2] * rho;
    }
}

namespace {

int nblk(long long n) { return (int)((n + 255) / 256); }

bool e3_setup(const bella_expl3d *a, Expl3Geom &G, Expl3Fields &F, AdvGeom &A, AdvFields &AF) {
    if (!a || a->inx < 5 || a->iny < 5 || a->inz < 5) return false;
    const double *req[] = {a->rho, a->rhou, a->rhov, a->rhow, a->rhoY, a->rhoX, a->S0n, a->hydro_rhoY0,
                           a->strat_inv};
    for (const double *p : req)
        if (!p) return false;
    G.icx = a->inx + 3; G.icy = a->iny + 3; G.icz = a->inz + 3;
    G.bc[0] = a->x_wall ? 1 : 0; G.bc[1] = a->y_wall ? 1 : 0; G.bc[2] = a->z_wall ? 1 : 0;
    G.dx = a->dx; G.dy = a->dy; G.dz = a->dz; G.dt = a->dt;
    G.Msq = a->Msq; G.g = a->g; G.gamm = a->gamm; G.nonhydro = a->nonhydro; G.compressibility = a->compressibility;
    for (int q = 0; q < 3; ++q) {
        G.cor[q] = a->coriolis[q];
        G.wind[q] = a->wind[q];
    }
    G.is_ArakawaKonor = a->is_ArakawaKonor;
    G.xsign = a->div_sign_2d ? 1.0 : -1.0;
    double *f[6] = {a->rho, a->rhou, a->rhov, a->rhow, a->rhoY, a->rhoX};
    for (int q = 0; q < 6; ++q) F.f[q] = AF.f[q] = f[q];
    A.nd = 3;
    A.ic[0] = G.icx; A.ic[1] = G.icy; A.ic[2] = G.icz;
    for (int q = 0; q < 3; ++q) A.bc[q] = G.bc[q];
    A.d[0] = a->dx; A.d[1] = a->dy; A.d[2] = a->dz;
    A.g = a->g; A.gamm = a->gamm; A.is_compressible = a->is_compressible;
    return true;
}

void e3_boundary(const AdvGeom &A, const AdvFields &AF, const bella_expl3d *a, cudaStream_t s) {
    for (int d = 0; d < 3; ++d) adv_boundary(A, d, AF, a->hydro_rhoY0, a->strat_inv, s);
}

}  // namespace
}  // namespace bella

using namespace bella;

extern "C" int bella_euler_forward3d(const bella_expl3d *a, void *stream) {
    Expl3Geom G;
    Expl3Fields F;
    AdvGeom A;
    AdvFields AF;
    if (!e3_setup(a, G, F, A, AF) || !a->p2 || !a->S0c || !a->scratch) return BELLA_EINVAL;
    cudaStream_t s = (cudaStream_t)stream;
    const long long nisc = (long long)(G.icx - 1) * (G.icy - 1) * (G.icz - 1);
    k_e3_zero_ghost<<<nblk((long long)G.icx * G.icz), 256, 0, s>>>(G, F);
    const Walk3 nodes = walk3(G.icx - 1, G.icy - 1, G.icz - 1, 1), cells = walk3(G.icx, G.icy, G.icz, 1);
    k_e3_fw_nodes<<<nodes.tiles.blocks, C3_THREADS, 0, s>>>(G, nodes, G.xsign * 0.25 / G.dx, 0.25 / G.dy, 0.25 / G.dz,
                                                    -G.dt * ((G.gamm - 1.0) / G.Msq) / 8.0, F, a->rhs_out, a->scratch);
    k_e3_fw_cells<<<cells.tiles.blocks, C3_THREADS, 0, s>>>(G, cells, F, a->p2, a->S0c, a->S0n);
    k_e3_fw_p2<<<nblk(nisc), 256, 0, s>>>(G, a->scratch, a->p2);
    const long long nn[3] = {(long long)G.icx + 1, (long long)G.icy + 1, (long long)G.icz + 1};
    for (int d = 0; d < 3; ++d)
        k_e3_ghost<<<nblk(nn[d == 0 ? 1 : 0] * nn[d == 2 ? 1 : 2]), 256, 0, s>>>(G, d, a->p2);
    e3_boundary(A, AF, a, s);
    return cudaGetLastError() == cudaSuccess ? BELLA_OK : BELLA_ECUDA;
}

extern "C" int bella_expl_part3d(const bella_expl3d *a, void *stream) {
    Expl3Geom G;
    Expl3Fields F;
    AdvGeom A;
    AdvFields AF;
    if (!e3_setup(a, G, F, A, AF)) return BELLA_EINVAL;
    cudaStream_t s = (cudaStream_t)stream;
    const Walk3 cells = walk3(G.icx, G.icy, G.icz, 0);
    k_e3_xp_cells<<<cells.tiles.blocks, C3_THREADS, 0, s>>>(G, cells, coriolis3(G.dt, G.nonhydro, G.cor), F, a->S0n);
    e3_boundary(A, AF, a, s);
    return cudaGetLastError() == cudaSuccess ? BELLA_OK : BELLA_ECUDA;
}
