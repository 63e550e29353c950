// bella_op2d.cu -- 2D 9-point nodal Helmholtz operator and the fused
// BiCGStab kernels built on it (sm_103a).
//
// The operator is the reference's lap2D_gather_new (laplacian.py:546-746)
// rewritten in cell-flux form: every cell c computes, from the diagonal
// differences d1 = BR - TL and d2 = TR - BL,
//   Gx = (d1 + d2)/2 = ((TR-TL)+(BR-BL))/2,  Gy = (d1 - d2)/2 = ((BL-TL)+(BR-TR))/2
//   Fx = Axx*Gx + Axy*Gy,  Fy = Ayy*Gy + Ayx*Gx,  P = Fx + Fy,  M = Fx - Fy
// once, and each node sums its four cells
//   y = dinv * ( (M[TR] - M[BL]) + (P[BR] - P[TL]) + hc*u )
//     = dinv * ( Fx[TR]+Fx[BR]-Fx[TL]-Fx[BL] + Fy[BL]+Fy[BR]-Fy[TL]-Fy[TR] + hc*u )
// which is algebraically the reference's Dxx+Dyy+Dyx+Dxy+hcenter*p scaled by
// diag_inv (laplacian.py:721-739); 9 additions per node instead of 13.  Walls are folded into the cell planes
// (zeroed outer cell column/row, laplacian.py:691-713); the periodic wrap
// with the duplicated seam (laplacian.py:595-638) is done on the halo load.
// The LAMB_BDRY variant (lap2D_numba_test with its padding and the kernel_9pt
// stencil, laplacian.py:531-543, 749-868) is the same operator on the same cell
// planes with a mirrored y boundary on the halo load and no cell zeroed.
//
// A warp marches a strip of nodes down the rows (bella_strip2d.cuh), computing the
// stencil input u on the fly from the Krylov vectors where the mode asks for it, and
// accumulates the inner products of the iteration in registers.
#include "bella_iter2d.cuh"

namespace bella {

// --------------------------------------------------------------------------
// operator packing: reference operands -> cell planes (FP64 and FP32)
// --------------------------------------------------------------------------
__global__ void k_pack2d_cells(bella_op2d op, double *a64, float *a32, dfloat *adf, int cross) {
    const int nx = op.nx, ny = op.ny;
    const size_t ncell = (size_t)(nx + 1) * (ny + 1);
    const double oodx = 1.0 / op.dx, oody = 1.0 / op.dy;
    for (size_t c = blockIdx.x * (size_t)blockDim.x + threadIdx.x; c < ncell;
         c += (size_t)gridDim.x * blockDim.x) {
        const int cj = (int)(c / (nx + 1)), ci = (int)(c - (size_t)cj * (nx + 1));
        double hx = op.hplusx[c], hy = op.hplusy[c];
        // wall handling: the outer cell column/row never couples (laplacian.py:691-713)
        if (op.x_wall && (ci == 0 || ci == nx)) { hx = 0.0; hy = 0.0; }
        if (op.y_wall == 1 && (cj == 0 || cj == ny)) { hx = 0.0; hy = 0.0; }   // not for the mirror (2)
        // with the half of Gx and Gy
        const double axx = 0.25 * oodx * oodx * op.cxx[c] * hx;
        const double ayy = 0.25 * oody * oody * op.cyy[c] * hy;
        const double axy = cross ? 0.25 * oodx * oody * (op.cxy ? op.cxy[c] : 0.0) * hy : 0.0;
        const double ayx = cross ? 0.25 * oodx * oody * (op.cyx ? op.cyx[c] : 0.0) * hx : 0.0;
        a64[c] = axx; a64[ncell + c] = ayy; a64[2 * ncell + c] = axy; a64[3 * ncell + c] = ayx;
        a32[c] = (float)axx; a32[ncell + c] = (float)ayy;
        a32[2 * ncell + c] = (float)axy; a32[3 * ncell + c] = (float)ayx;
        if (adf) {   // double-float planes (absent in the allocation-free path)
            adf[c] = dfloat(axx); adf[ncell + c] = dfloat(ayy);
            adf[2 * ncell + c] = dfloat(axy); adf[3 * ncell + c] = dfloat(ayx);
        }
    }
}

// node planes; z = left null weights / diag_inv (trapezoid weight 1/2 on the
// duplicated periodic seam), used to project the pseudo-incompressible
// solution onto the operator's range.
__global__ void k_pack2d_nodes(bella_op2d op, double *dinv64, float *dinv32, double *hc64,
                               float *hc32, double *z64, dfloat *dinvdf, dfloat *hcdf) {
    const int nx = op.nx, ny = op.ny;
    const size_t n = (size_t)nx * ny;
    for (size_t g = blockIdx.x * (size_t)blockDim.x + threadIdx.x; g < n;
         g += (size_t)gridDim.x * blockDim.x) {
        const int j = (int)(g / nx), i = (int)(g - (size_t)j * nx);
        const double d = op.diag_inv[g];
        const double h = op.hcenter ? op.hcenter[g] : 0.0;
        dinv64[g] = d; dinv32[g] = (float)d;
        hc64[g] = h;   hc32[g] = (float)h;
        if (dinvdf) { dinvdf[g] = dfloat(d); hcdf[g] = dfloat(h); }
        double w = 1.0;
        if (!op.x_wall && (i == 0 || i == nx - 1)) w *= 0.5;
        if (op.y_wall == 0 && (j == 0 || j == ny - 1)) w *= 0.5;
        z64[g] = w / d;
    }
}

// --------------------------------------------------------------------------
// fused stencil kernel: a warp per strip (bella_strip2d.cuh), strips of h rows shared out
// evenly; the inner products are accumulated in registers (double-float for FP32 types)
// --------------------------------------------------------------------------
// CTAs per SM: 64 registers a thread, 128 for the pairs of double-floats
template <typename T> constexpr int stencil_blocks() { return Lane<T>::N == 2 ? 2 : 4; }

template <typename T, int MODE, bool CROSS, bool HC>
__global__ void __launch_bounds__(NTHREADS, stencil_blocks<T>())
k_stencil2d(Op2D<T> op, StArgs<T> a, int h, KState *ks, double *partials, unsigned *counter) {
    int iter = 0;
    T alpha = 0, beta = 0, omega = 0;
    if (MODE == M_PDIR || MODE == M_SDIR) {
        if (ks->done) return;
        iter = ks->iter;
        alpha = (T)ks->alpha;
        beta = (T)ks->beta;
        omega = (T)ks->omega;
    }
    typename LaneAcc<T>::type acc0, acc1, acc2;
    acc0.zero(); acc1.zero(); acc2.zero();
    // strip after strip to block after block: every SM gets its share whatever their number
    const int warp = (threadIdx.x >> 5) * gridDim.x + blockIdx.x, nwarps = gridDim.x * (NTHREADS / 32);
    const int strips = strips_across(op.nx, strip_width<T>()) * strips_down(op.ny, h);
    stencil_phase<T, MODE, CROSS, HC, false>(op, a, h, iter, alpha, beta, omega, warp, strips, nwarps, acc0, acc1, acc2);
    if (MODE == M_APPLY) return;

    double v[3] = {acc0.value(), acc1.value(), acc2.value()};
    double tot[3];
    if (!grid_sum<3>(v, partials, counter, tot)) return;
    if (threadIdx.x != 0) return;
    if (MODE == M_RESID) {
        ks->dot_aux2 = tot[0];
    } else if (MODE == M_PDIR) {
        finalize_pdir(ks, tot[0]);
    } else {
        finalize_sdir(ks, tot[0], tot[1], tot[2]);
    }
}

// Whole BiCGStab iterations, `iters` of them or until the state is done, in one cooperative
// launch: one block per SM, the three phases of an iteration separated by the sums over the grid
// that they need anyway (grid_totals), the scalars derived by every block alike from the same
// sums (finalize_*).  A kernel per phase costs 13 us an iteration and phase whatever its
// work -- its launch, the last-block reduction and the state's way through memory -- which
// is the whole time of a small grid.  161x81 nodes, FP64: 47 -> 23 us an iteration, in small blocks 21
// (of which three sums 11); 1001x500 and 2049x1025, double-float: 73 -> 45 and 157 -> 97 us.
template <typename T> __host__ __device__ constexpr int iter2d_threads() { return sizeof(T) == 4 ? 1024 : 512; }   // 64 or 128 registers

template <typename T, bool CROSS, bool HC, bool VEC>
__global__ void __launch_bounds__(iter2d_threads<T>(), 1)
k_iter2d(Op2D<T> op, StArgs<T> a, T *x, T *r, long long n, int h, int iters, KState *ks, SumWord *words) {
    __shared__ KState k;
    __shared__ double tot[3];
    __shared__ SumShared sums;
    const int t = threadIdx.x, warp = (t >> 5) * gridDim.x + blockIdx.x, nwarps = gridDim.x * (blockDim.x >> 5);
    if (t == 0) k = *ks;
    __syncthreads();
    // warps of this block that have strips, and pairs of elements
    const int strips = strips_across(op.nx, strip_width<T>()) * strips_down(op.ny, h);
    const long long pairs = (n / 2 + 31) / 32 + 1;
    auto active = [&](long long items) {
        const long long w = (items - blockIdx.x + gridDim.x - 1) / gridDim.x;
        return (int)(w < 1 ? 1 : w < (blockDim.x >> 5) ? w : (blockDim.x >> 5));
    };
    const int act_s = active(strips), act_u = active(pairs);
    unsigned long long seq = 0;
    // thread 0 takes the step that needs the totals, or ends the solve when they did not arrive
    auto step = [&](bool ok, auto finalize) {
        if (t == 0) {
            if (ok) {
                finalize();
            } else {
                k.done = 1;
                k.status = BELLA_ECUDA;
            }
        }
        __syncthreads();
    };
    for (int q = 0; q < iters && !k.done; ++q) {
        typename LaneAcc<T>::type c0, c1, c2;
        {
            c0.zero(); c1.zero(); c2.zero();
            stencil_phase<T, M_PDIR, CROSS, HC, true>(op, a, h, k.iter, (T)k.alpha, (T)k.beta, (T)k.omega, warp, strips, nwarps,
                                                      c0, c1, c2);
            double v[1] = {c0.value()};
            const bool ok = grid_totals<1>(v, act_s, words, ++seq, sums, tot);
            step(ok, [&] { finalize_pdir(&k, tot[0]); });
            if (k.done) break;
        }
        {
            c0.zero(); c1.zero(); c2.zero();
            stencil_phase<T, M_SDIR, CROSS, HC, true>(op, a, h, k.iter, (T)k.alpha, (T)k.beta, (T)k.omega, warp, strips, nwarps,
                                                      c0, c1, c2);
            double v[3] = {c0.value(), c1.value(), c2.value()};
            const bool ok = grid_totals<3>(v, act_s, words, ++seq, sums, tot);
            step(ok, [&] { finalize_sdir(&k, tot[0], tot[1], tot[2]); });
            if (k.done) break;
        }
        typename Acc<T>::type u0, u1;
        u0.zero(); u1.zero();
        const bool odd = k.iter & 1;                   // p and v written by this iteration's first phase
        update_phase<T, VEC, true>(n, x, odd ? a.p0 : a.p1, r, odd ? a.v0 : a.v1, a.y, a.rh, (T)k.alpha, (T)k.omega,
                                   k.early != 0, warp * 32LL + (t & 31), nwarps * 32LL, u0, u1);
        double v[2] = {u0.value(), u1.value()};
        const bool ok = grid_totals<2>(v, act_u, words, ++seq, sums, tot);
        // the two quotients of beta by two lanes, in one division's time
        double quot = t == 0 ? tot[0] / k.rho : t == 1 ? k.alpha / k.omega : 0.0;
        if (t < 32) quot *= __shfl_down_sync(0xffffffffu, quot, 1);
        step(ok, [&] { finalize_update(&k, tot[0], tot[1], quot); });
    }
    // a block that gave up stops the others' next sum, block 0's too
    if (blockIdx.x == 0 && t == 0) *ks = k;
}

// The same iterations, to the same bits, in smaller blocks of which two fit an SM, so that solves on other
// streams run beside it: a block of k_iter2d takes an SM for itself, and solves then come one after
// the other, where those of a kernel a phase had overlapped.  Block p does the work of nv (1, 2 or 4) of
// k_iter2d's G blocks, one for every SM; the sums keep k_iter2d's order.  Solves of 64 iterations, us a solve for
// 1, 4 and 8 host threads, k_iter2d | this | a kernel a phase:
//   FP64          161x81   1563 1476 1482 | 1456  437  415 | 3143  834  492
//                 225x113  1597 1518 1506 | 1587  882  867 | 3199  877  566
//                 449x225  2079 1976 1966 | 2075 1181 1175 | 3338 1405 1055
//   double-float  161x81   1858 1697 1694 | 1795  492  326 | 2972  833  493
//                 321x161  1961 1804 1784 | 1803  993  978 | 3133  949  602
// Three blocks an SM (80 registers) take eight threads' 225x113 to 659, but one's to 1673.
constexpr int FEW_PER_SM = 2;                          // 128 registers

template <typename T, bool CROSS, bool HC, bool VEC>
__global__ void __launch_bounds__(32 * FEW_WARPS, FEW_PER_SM)
k_iter2d_few(Op2D<T> op, StArgs<T> a, T *x, T *r, long long n, int h, int iters, int G, int nv, KState *ks,
             SumWord *words) {
    constexpr int FULL = iter2d_threads<T>() / 32;     // k_iter2d's warps
    __shared__ KState k;
    __shared__ double tot[3];
    __shared__ SumSharedFew<FULL> sums;
    const int t = threadIdx.x, lane = t & 31, wid = t >> 5;
    // which of the nv blocks this warp works for, and as which of its warps
    const int block = blockIdx.x + wid % nv * gridDim.x, row = wid / nv, nwarps = G * FULL;
    const bool on = block < G;
    if (t == 0) k = *ks;
    __syncthreads();
    const int strips = strips_across(op.nx, strip_width<T>()) * strips_down(op.ny, h);
    const long long pairs = (n / 2 + 31) / 32 + 1;
    // rows of warps that have strips, or pairs of elements
    const int rows_s = (strips + G - 1) / G, rows_u = pairs < (long long)FULL * G ? (int)((pairs + G - 1) / G) : FULL;
    // the words of `items` strips, or of 32 pairs of elements each
    auto words_of = [&](long long items) { return items < (int)gridDim.x ? (int)gridDim.x : items < G ? (int)items : G; };
    unsigned long long seq = 0;
    auto step = [&](bool ok, auto finalize) {
        if (t == 0) {
            if (ok) {
                finalize();
            } else {
                k.done = 1;
                k.status = BELLA_ECUDA;
            }
        }
        __syncthreads();
    };
    for (int q = 0; q < iters && !k.done; ++q) {
        typename LaneAcc<T>::type c0, c1, c2;
        c0.zero(); c1.zero(); c2.zero();
        const int first = on ? row * G + block : strips;           // every strip has a warp
        stencil_phase<T, M_PDIR, CROSS, HC, true>(op, a, h, k.iter, (T)k.alpha, (T)k.beta, (T)k.omega, first, strips, nwarps,
                                                  c0, c1, c2);
        sums.sm[0][t] = c0.value();
        bool ok = grid_totals_few<1>(nv, rows_s, words_of(strips), words, ++seq, sums, tot);
        step(ok, [&] { finalize_pdir(&k, tot[0]); });
        if (k.done) break;
        c0.zero(); c1.zero(); c2.zero();
        stencil_phase<T, M_SDIR, CROSS, HC, true>(op, a, h, k.iter, (T)k.alpha, (T)k.beta, (T)k.omega, first, strips, nwarps,
                                                  c0, c1, c2);
        sums.sm[0][t] = c0.value();
        sums.sm[1][t] = c1.value();
        sums.sm[2][t] = c2.value();
        ok = grid_totals_few<3>(nv, rows_s, words_of(strips), words, ++seq, sums, tot);
        step(ok, [&] { finalize_sdir(&k, tot[0], tot[1], tot[2]); });
        if (k.done) break;
        const bool odd = k.iter & 1;                   // p and v written by this iteration's first phase
        T *const p = odd ? a.p0 : a.p1, *const v = odd ? a.v0 : a.v1;
        const long long warp = on ? row * (long long)G + block : pairs;
        typename Acc<T>::type u0[2], u1[2];
        if (rows_u <= FEW_WARPS) {
            u0[0].zero(); u1[0].zero();
            update_phase<T, VEC, true>(n, x, p, r, v, a.y, a.rh, (T)k.alpha, (T)k.omega, k.early != 0, warp * 32 + lane,
                                       nwarps * 32LL, u0[0], u1[0]);
            sums.sm[0][t] = u0[0].value();
            sums.sm[1][t] = u1[0].value();
        } else {                                       // nv = 1: the shares of two warps at a time
            for (int j = 0; j < rows_u; j += 2 * FEW_WARPS) {
                u0[0].zero(); u1[0].zero(); u0[1].zero(); u1[1].zero();
                const long long f = (warp + (long long)j * G) * 32 + lane;
                update_two<T, VEC, true>(n, x, p, r, v, a.y, a.rh, (T)k.alpha, (T)k.omega, k.early != 0, f,
                                         f + 32LL * FEW_WARPS * G, nwarps * 32LL, u0, u1);
#pragma unroll
                for (int q = 0; q < 2; ++q) {
                    sums.sm[0][t + 32 * (j + q * FEW_WARPS)] = u0[q].value();
                    sums.sm[1][t + 32 * (j + q * FEW_WARPS)] = u1[q].value();
                }
            }
        }
        ok = grid_totals_few<2>(nv, rows_u, words_of(pairs), words, ++seq, sums, tot);
        double quot = t == 0 ? tot[0] / k.rho : t == 1 ? k.alpha / k.omega : 0.0;
        if (t < 32) quot *= __shfl_down_sync(0xffffffffu, quot, 1);
        step(ok, [&] { finalize_update(&k, tot[0], tot[1], quot); });
    }
    if (blockIdx.x == 0 && t == 0) *ks = k;
}

// --------------------------------------------------------------------------
// host launchers
// --------------------------------------------------------------------------
template <typename T>
static Op2D<T> make_op(bella_ws *ws);

template <>
Op2D<double> make_op<double>(bella_ws *ws) {
    const size_t nc = (size_t)(ws->nx + 1) * (ws->ny + 1);
    Op2D<double> o;
    o.nx = ws->nx; o.ny = ws->ny; o.ymirror = ws->ymirror;
    o.axx = ws->a64; o.ayy = ws->a64 + nc; o.axy = ws->a64 + 2 * nc; o.ayx = ws->a64 + 3 * nc;
    o.dinv = ws->dinv64; o.hc = ws->hc64;
    return o;
}

template <>
Op2D<dfloat> make_op<dfloat>(bella_ws *ws) {
    const size_t nc = (size_t)(ws->nx + 1) * (ws->ny + 1);
    Op2D<dfloat> o;
    o.nx = ws->nx; o.ny = ws->ny; o.ymirror = ws->ymirror;
    o.axx = ws->adf; o.ayy = ws->adf + nc; o.axy = ws->adf + 2 * nc; o.ayx = ws->adf + 3 * nc;
    o.dinv = ws->dinvdf; o.hc = ws->hcdf;
    return o;
}

template <>
Op2D<float> make_op<float>(bella_ws *ws) {
    const size_t nc = (size_t)(ws->nx + 1) * (ws->ny + 1);
    Op2D<float> o;
    o.nx = ws->nx; o.ny = ws->ny; o.ymirror = ws->ymirror;
    o.axx = ws->a32; o.ayy = ws->a32 + nc; o.axy = ws->a32 + 2 * nc; o.ayx = ws->a32 + 3 * nc;
    o.dinv = ws->dinv32; o.hc = ws->hc32;
    return o;
}

constexpr int STENCIL_WARPS = NTHREADS / 32;

template <typename T, int MODE>
static void launch_mode(bella_ws *ws, const StArgs<T> &a, cudaStream_t s) {
    Op2D<T> op = make_op<T>(ws);
    // one resident wave at most (partials hold MAXGRID CTAs), a block for every strip while there are
    // SMs without one
    const int sms = num_sms(), per_sm = stencil_blocks<T>();
    const int h = strip_height<T>(ws->nx, ws->ny, sms, per_sm * STENCIL_WARPS);
    const long long strips = (long long)strips_across(ws->nx, strip_width<T>()) * strips_down(ws->ny, h);
    const int grid = strips < (long long)sms * per_sm ? (int)strips : sms * per_sm, blk = NTHREADS;
    const int pk = MODE == M_PDIR ? PK_PDIR : MODE == M_SDIR ? PK_SDIR : MODE == M_RESID ? PK_RESID : -1;
    if (pk >= 0) prof_begin(ws, pk, s);
    if (ws->cross) {
        if (ws->has_hc) k_stencil2d<T, MODE, true, true><<<grid, blk, 0, s>>>(op, a, h, ws->ks, ws->partials, ws->counter);
        else            k_stencil2d<T, MODE, true, false><<<grid, blk, 0, s>>>(op, a, h, ws->ks, ws->partials, ws->counter);
    } else {
        if (ws->has_hc) k_stencil2d<T, MODE, false, true><<<grid, blk, 0, s>>>(op, a, h, ws->ks, ws->partials, ws->counter);
        else            k_stencil2d<T, MODE, false, false><<<grid, blk, 0, s>>>(op, a, h, ws->ks, ws->partials, ws->counter);
    }
    if (pk >= 0) prof_end(ws, pk, s);
    ws->launches++;
}

int op2d_pack(bella_ws *ws, const bella_op2d *op, cudaStream_t s) {
    const size_t ncell = (size_t)(op->nx + 1) * (op->ny + 1);
    int g = (int)((ncell + 255) / 256);
    if (g > num_sms() * 8) g = num_sms() * 8;
    k_pack2d_cells<<<g, 256, 0, s>>>(*op, ws->a64, ws->a32, ws->adf, ws->cross);
    k_pack2d_nodes<<<g, 256, 0, s>>>(*op, ws->dinv64, ws->dinv32, ws->hc64, ws->hc32, ws->z64, ws->dinvdf,
                                     ws->hcdf);
    ws->launches += 2;
    return cudaGetLastError() == cudaSuccess ? BELLA_OK : BELLA_ECUDA;
}

void op2d_apply(bella_ws *ws, int prec, const void *x, void *y, cudaStream_t s) {
    if (prec == 0) {
        StArgs<double> a = {};
        a.x = (const double *)x; a.y = (double *)y;
        launch_mode<double, M_APPLY>(ws, a, s);
    } else {
        StArgs<float> a = {};
        a.x = (const float *)x; a.y = (float *)y;
        launch_mode<float, M_APPLY>(ws, a, s);
    }
}

void op2d_resid(bella_ws *ws, int prec, const void *x, const void *b, void *r, cudaStream_t s) {
    if (prec == 0) {
        StArgs<double> a = {};
        a.x = (const double *)x; a.b = (const double *)b; a.y = (double *)r;
        launch_mode<double, M_RESID>(ws, a, s);
    } else {
        StArgs<float> a = {};
        a.x = (const float *)x; a.b = (const float *)b; a.y = (float *)r;
        launch_mode<float, M_RESID>(ws, a, s);
    }
}

static StArgs<dfloat> iter_args(bella_ws *ws, dfloat) {
    StArgs<dfloat> a = {};
    a.r = ws->rdf; a.rh = ws->rhdf; a.y = ws->tdf;
    a.p0 = ws->pdf[0]; a.p1 = ws->pdf[1]; a.v0 = ws->vdf[0]; a.v1 = ws->vdf[1];
    return a;
}
static StArgs<double> iter_args(bella_ws *ws, double) {
    StArgs<double> a = {};
    a.r = ws->r64k; a.rh = ws->rh64; a.y = ws->t64;
    a.p0 = ws->p64[0]; a.p1 = ws->p64[1]; a.v0 = ws->v64[0]; a.v1 = ws->v64[1];
    return a;
}
static StArgs<float> iter_args(bella_ws *ws, float) {
    StArgs<float> a = {};
    a.r = ws->r32; a.rh = ws->rh32; a.y = ws->t32;
    a.p0 = ws->p32[0]; a.p1 = ws->p32[1]; a.v0 = ws->v32[0]; a.v1 = ws->v32[1];
    return a;
}

// one BiCGStab iteration in three launches: PDIR stencil, SDIR stencil, vector update
template <typename T>
static void iterate_launches(bella_ws *ws, cudaStream_t s) {
    const StArgs<T> a = iter_args(ws, T());
    launch_mode<T, M_PDIR>(ws, a, s);
    launch_mode<T, M_SDIR>(ws, a, s);
    launch_update<T>(ws, s);
}

// k_iter2d's blocks that one of k_iter2d_few's does the work of; 0: k_iter2d.  As many as leave each SM
// quarter one strip, since its FP64 arithmetic is what two would wait for, and every strip a warp; with
// nv above 1 every 32 pairs of elements too.
static int few_blocks(long long strips, long long n, int sms) {
    const long long rows_s = (strips + sms - 1) / sms, rows_u = ((n / 2 + 31) / 32 + sms) / sms;
    for (int nv = 4; nv >= 2; nv /= 2)
        if (rows_s * nv <= 4 && rows_u * nv <= FEW_WARPS) return nv;
    return rows_s <= FEW_WARPS ? 1 : 0;
}

template <typename T, bool CROSS, bool HC>
static const void *iter2d_kernel(bool few, bool vec) {
    if (few) return vec ? (const void *)k_iter2d_few<T, CROSS, HC, true> : (const void *)k_iter2d_few<T, CROSS, HC, false>;
    return vec ? (const void *)k_iter2d<T, CROSS, HC, true> : (const void *)k_iter2d<T, CROSS, HC, false>;
}

// `iters` iterations in one cooperative launch; BELLA_ENOOP: the device cannot hold it
template <typename T>
static int iterate_coop(bella_ws *ws, T *x, int iters, cudaStream_t s) {
    const StArgs<T> a = iter_args(ws, T());
    T *r = const_cast<T *>(a.r);
    const bool vec = reinterpret_cast<uintptr_t>(x) % 16 == 0;      // x may be the caller's; the others are aligned
    const int sms = num_sms(), h = strip_height<T>(ws->nx, ws->ny, sms, iter2d_threads<T>() / 32);
    const long long strips = (long long)strips_across(ws->nx, strip_width<T>()) * strips_down(ws->ny, h);
    const int few = few_blocks(strips, ws->n, sms), threads = few ? 32 * FEW_WARPS : iter2d_threads<T>();
    const void *k = ws->cross ? (ws->has_hc ? iter2d_kernel<T, true, true>(few, vec) : iter2d_kernel<T, true, false>(few, vec))
                              : (ws->has_hc ? iter2d_kernel<T, false, true>(few, vec) : iter2d_kernel<T, false, false>(few, vec));
    int per_sm = 0;
    if (cudaOccupancyMaxActiveBlocksPerMultiprocessor(&per_sm, k, threads, 0) != cudaSuccess || per_sm < 1)
        return BELLA_ENOOP;
    Op2D<T> op = make_op<T>(ws);
    StArgs<T> args_a = a;
    long long n = ws->n;
    int hh = h, it = iters, G = sms, nv = few;
    SumWord *words = reinterpret_cast<SumWord *>(ws->partials);        // in the reduction partials' buffer
    static_assert(SUM_WORDS * sizeof(SumWord) <= sizeof(double) * NQ * MAXGRID, "the sums' words fit the partials");
    if (cudaMemsetAsync(words, 0, SUM_WORDS * sizeof(SumWord), s) != cudaSuccess) return BELLA_ECUDA;
    void *args_full[] = {&op, &args_a, &x, &r, &n, &hh, &it, &ws->ks, &words};
    void *args_few[] = {&op, &args_a, &x, &r, &n, &hh, &it, &G, &nv, &ws->ks, &words};
    const cudaError_t rc = cudaLaunchCooperativeKernel(k, few ? (sms + few - 1) / few : sms, threads,
                                                       few ? args_few : args_full, 0, s);
    if (rc == cudaErrorCooperativeLaunchTooLarge) {    // the stream's context has a part of the SMs only
        cudaGetLastError();
        return BELLA_ENOOP;
    }
    if (rc != cudaSuccess) return BELLA_ECUDA;
    ws->launches++;
    return BELLA_OK;
}

// BiCGStab iterations until the state is done, `iters` at most.  prec: 0 FP64, 1 FP32, 2 double-float
int op2d_iterations(bella_ws *ws, int prec, int iters, cudaStream_t s) {
    int rc = BELLA_ENOOP;
    if (!ws->prof) {                                   // per-kernel times need a kernel per phase
        if (prec == 2) rc = iterate_coop<dfloat>(ws, ws->xdf, iters, s);
        else if (prec == 0) rc = iterate_coop<double>(ws, ws->x64v, iters, s);
        else rc = iterate_coop<float>(ws, ws->x32, iters, s);
    }
    if (rc != BELLA_ENOOP) return rc;
    for (int k = 0; k < iters; ++k) {
        if (prec == 2) iterate_launches<dfloat>(ws, s);
        else if (prec == 0) iterate_launches<double>(ws, s);
        else iterate_launches<float>(ws, s);
    }
    return BELLA_OK;
}

}  // namespace bella
