// bella_iter2d.cuh -- the three phases of a BiCGStab iteration on the 2D operator as device
// functions, for the kernels that run one phase each (bella_op2d.cu, bella_krylov.cu) and the one
// that runs whole iterations (k_iter2d, bella_op2d.cu).
#pragma once
#include "bella_strip2d.cuh"

namespace bella {

template <typename T>
struct StArgs {
    const T *x;      // APPLY / RESID input
    const T *b;      // RESID right-hand side
    T *y;            // APPLY / RESID / SDIR output
    const T *r, *rh;
    T *p0, *p1, *v0, *v1;
};

// The operator in one of its modes over this warp's strips (first, first + step, ... below end); the
// iteration's scalars for M_PDIR (p = r + beta (p - omega v), v = A p, <r^, v>) and M_SDIR (s = r -
// alpha v, t = A s, <t,s>, <t,t>, <s,s>), RESID: ||b - A x||^2 in acc0.  CG: the Krylov vectors
// are written by other blocks of the same launch.
template <typename T, int MODE, bool CROSS, bool HC, bool CG>
__device__ __forceinline__ void stencil_phase(const Op2D<T> &op, const StArgs<T> &a, int h, int iter, T alpha, T beta,
                                              T omega, int first_strip, int end_strip, int step,
                                              typename LaneAcc<T>::type &acc0, typename LaneAcc<T>::type &acc1,
                                              typename LaneAcc<T>::type &acc2) {
    typedef Lane<T> LN;
    typedef typename LN::V V;
    constexpr int N = LN::N;
    struct Q { T r, p, v; };
    struct Q2 { T a; };
    const int par = iter & 1;
    const bool first = iter == 0;
    const V va = LN::splat(alpha), vb = LN::splat(beta), vo = LN::splat(omega);
    const T *pin = par ? a.p1 : a.p0;
    T *pout = par ? a.p0 : a.p1;
    const T *vold = par ? a.v1 : a.v0;
    T *vnew = par ? a.v0 : a.v1;
    const T *vin = (MODE == M_PDIR) ? vold : vnew;   // SDIR reads the fresh v
    T *yout = (MODE == M_PDIR) ? vnew : a.y;
    const int across = strips_across(op.nx, strip_width<T>());
    auto join = [](const Q (&q)[N], T Q::*m) {
        T t[N];
#pragma unroll
        for (int n = 0; n < N; ++n) t[n] = q[n].*m;
        return LN::join(t);
    };
    for (int st = first_strip; st < end_strip; st += step) {
        const int sy = st / across, sx = st - sy * across;
        march_strip<T, CROSS, HC, Q, Q2>(op, sx, sy, h,
            [&](unsigned g, Q &q) {
                if (MODE == M_APPLY || MODE == M_RESID) {
                    q.r = a.x[g];
                } else {
                    q.r = ld_vec<CG>(a.r + g);
                    q.v = ld_vec<CG>(vin + g);
                    if (MODE == M_PDIR) q.p = ld_vec<CG>(pin + g);
                }
            },
            [&](const Q (&q)[N]) {
                const V r = join(q, &Q::r);
                if (MODE == M_PDIR) return first ? r : r + vb * (join(q, &Q::p) - vo * join(q, &Q::v));
                if (MODE == M_SDIR) return r - va * join(q, &Q::v);
                return r;
            },
            [&](unsigned g, T u) { if (MODE == M_PDIR) pout[g] = u; },
            [&](unsigned g, Q2 &q) {
                if (MODE == M_RESID) q.a = a.b[g];
                else if (MODE == M_PDIR) q.a = a.rh[g];
            },
            [&](const Q2 (&q)[N], V u, V yv, const unsigned (&g)[N], const bool (&on)[N]) {
                T t[N], w[N], x[N];
#pragma unroll
                for (int n = 0; n < N; ++n) t[n] = on[n] ? q[n].a : (T)0;
                if (MODE == M_RESID) yv = LN::join(t) - yv;
                LN::split(yv, w);
#pragma unroll
                for (int n = 0; n < N; ++n)
                    if (on[n]) yout[g[n]] = w[n];
                if (MODE == M_APPLY) return;
                // the columns that are not owned add zeros
                LN::split(u, x);
#pragma unroll
                for (int n = 0; n < N; ++n)
                    if (!on[n]) { w[n] = (T)0; x[n] = (T)0; }
                yv = LN::join(w);
                if (MODE == M_RESID) {
                    acc0.add_prod(yv, yv);
                } else if (MODE == M_PDIR) {
                    acc0.add_prod(LN::join(t), yv);
                } else {
                    u = LN::join(x);
                    acc0.add_prod(yv, u);
                    acc1.add_prod(yv, yv);
                    acc2.add_prod(u, u);
                }
            });
    }
}

// two neighbouring elements, as one 16-byte access where VEC (double-float and FP64; 8 bytes FP32)
template <bool CG> __device__ __forceinline__ void load_two(const double *p, double (&a)[2]) {
    const double2 q = CG ? __ldcg(reinterpret_cast<const double2 *>(p)) : *reinterpret_cast<const double2 *>(p);
    a[0] = q.x; a[1] = q.y;
}
template <bool CG> __device__ __forceinline__ void load_two(const float *p, float (&a)[2]) {
    const float2 q = CG ? __ldcg(reinterpret_cast<const float2 *>(p)) : *reinterpret_cast<const float2 *>(p);
    a[0] = q.x; a[1] = q.y;
}
template <bool CG> __device__ __forceinline__ void load_two(const dfloat *p, dfloat (&a)[2]) {
    const float4 q = CG ? __ldcg(reinterpret_cast<const float4 *>(p)) : *reinterpret_cast<const float4 *>(p);
    a[0] = dfloat(q.x, q.y); a[1] = dfloat(q.z, q.w);
}
__device__ __forceinline__ void store_two(double *p, const double (&a)[2]) {
    *reinterpret_cast<double2 *>(p) = make_double2(a[0], a[1]);
}
__device__ __forceinline__ void store_two(float *p, const float (&a)[2]) {
    *reinterpret_cast<float2 *>(p) = make_float2(a[0], a[1]);
}
__device__ __forceinline__ void store_two(dfloat *p, const dfloat (&a)[2]) {
    *reinterpret_cast<float4 *>(p) = make_float4(a[0].hi, a[0].lo, a[1].hi, a[1].lo);
}
template <typename T, bool VEC, bool CG>
__device__ __forceinline__ void load_pair(const T *p, T (&a)[2]) {
    if (VEC) {
        load_two<CG>(p, a);
    } else {
        a[0] = ld_vec<CG>(p);
        a[1] = ld_vec<CG>(p + 1);
    }
}
template <typename T, bool VEC>
__device__ __forceinline__ void store_pair(T *p, const T (&a)[2]) {
    if (VEC) {
        store_two(p, a);
    } else {
        p[0] = a[0];
        p[1] = a[1];
    }
}

// x += alpha p + omega s,  r = s - omega t  (s = r - alpha v recomputed), with <r^, r> and
// ||r||^2 of the new residual; two neighbouring elements a thread and step, this thread's
// pairs first, first + step, ...  VEC: every vector 16-byte aligned.
template <typename T, bool VEC, bool CG>
__device__ __forceinline__ void update_phase(long long n, T *__restrict__ x, const T *__restrict__ p, T *__restrict__ r,
                                             const T *__restrict__ v, const T *__restrict__ t,
                                             const T *__restrict__ rh, T alpha, T omega, bool early, long long first,
                                             long long step, typename Acc<T>::type &a0, typename Acc<T>::type &a1) {
    auto one = [&](T &xg, T pg, T &rg, T vg, T tg, T hg) {
        if (early) {
            xg = xg + alpha * pg;
            return;
        }
        const T s = rg - alpha * vg;
        xg = xg + (alpha * pg + omega * s);
        rg = s - omega * tg;
        a0.add_prod(hg, rg);
        a1.add_prod(rg, rg);
    };
    const long long n2 = n / 2;
    for (long long i = first; i < n2; i += step) {
        T xg[2], pg[2], rg[2], vg[2], tg[2], hg[2];
        load_pair<T, VEC, CG>(x + 2 * i, xg);
        load_pair<T, VEC, CG>(p + 2 * i, pg);
        load_pair<T, VEC, CG>(r + 2 * i, rg);
        load_pair<T, VEC, CG>(v + 2 * i, vg);
        load_pair<T, VEC, CG>(t + 2 * i, tg);
        load_pair<T, VEC, false>(rh + 2 * i, hg);
#pragma unroll
        for (int q = 0; q < 2; ++q) one(xg[q], pg[q], rg[q], vg[q], tg[q], hg[q]);
        store_pair<T, VEC>(x + 2 * i, xg);
        if (!early) store_pair<T, VEC>(r + 2 * i, rg);
    }
    if ((n & 1) && first == 0) {
        T xg = ld_vec<CG>(x + n - 1), rg = ld_vec<CG>(r + n - 1);
        one(xg, ld_vec<CG>(p + n - 1), rg, ld_vec<CG>(v + n - 1), ld_vec<CG>(t + n - 1), rh[n - 1]);
        x[n - 1] = xg;
        r[n - 1] = rg;
    }
}

// The same for two threads of that numbering at once, first and second (the later one), with the
// loads of both in flight together and sums for each.
template <typename T, bool VEC, bool CG>
__device__ __forceinline__ void update_two(long long n, T *__restrict__ x, const T *__restrict__ p, T *__restrict__ r,
                                           const T *__restrict__ v, const T *__restrict__ t, const T *__restrict__ rh,
                                           T alpha, T omega, bool early, long long first, long long second,
                                           long long step, typename Acc<T>::type (&a0)[2], typename Acc<T>::type (&a1)[2]) {
    auto one = [&](T &xg, T pg, T &rg, T vg, T tg, T hg, int k) {
        if (early) {
            xg = xg + alpha * pg;
            return;
        }
        const T s = rg - alpha * vg;
        xg = xg + (alpha * pg + omega * s);
        rg = s - omega * tg;
        a0[k].add_prod(hg, rg);
        a1[k].add_prod(rg, rg);
    };
    const long long n2 = n / 2;
    const bool last = (n & 1) && first == 0;           // this thread also has the odd element
    for (; first < n2; first += step, second += step) {
        const bool both = second < n2;
        const long long at[2] = {first, both ? second : first};
        T xg[2][2], pg[2][2], rg[2][2], vg[2][2], tg[2][2], hg[2][2];
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            load_pair<T, VEC, CG>(x + 2 * at[k], xg[k]);
            load_pair<T, VEC, CG>(p + 2 * at[k], pg[k]);
            load_pair<T, VEC, CG>(r + 2 * at[k], rg[k]);
            load_pair<T, VEC, CG>(v + 2 * at[k], vg[k]);
            load_pair<T, VEC, CG>(t + 2 * at[k], tg[k]);
            load_pair<T, VEC, false>(rh + 2 * at[k], hg[k]);
        }
#pragma unroll
        for (int k = 0; k < 2; ++k) {
            if (k && !both) break;
#pragma unroll
            for (int q = 0; q < 2; ++q) one(xg[k][q], pg[k][q], rg[k][q], vg[k][q], tg[k][q], hg[k][q], k);
            store_pair<T, VEC>(x + 2 * at[k], xg[k]);
            if (!early) store_pair<T, VEC>(r + 2 * at[k], rg[k]);
        }
    }
    if (last) {
        T xg = ld_vec<CG>(x + n - 1), rg = ld_vec<CG>(r + n - 1);
        one(xg, ld_vec<CG>(p + n - 1), rg, ld_vec<CG>(v + n - 1), ld_vec<CG>(t + n - 1), rh[n - 1], 0);
        x[n - 1] = xg;
        r[n - 1] = rg;
    }
}

// ---- sums over all blocks of a cooperative launch ---------------------------------------
// Each block publishes its sums and reads everybody's, which also is the grid's barrier: what a
// block wrote before is seen by all after.  A value and the number of the sum it belongs
// to are one 16-byte word, written and read as one (b128), so that a reader needs neither a
// flag nor a second load.  Two sets of words take turns (seq's parity): a block can publish
// sum seq + 2 only after every block has published seq + 1, that is, has read all of seq.
//
// What it costs is latency: an FP64 addition 65 clocks, which also is its unit's rate (one per
// SM quarter, half a lane a clock), a fence 900, a round trip to L2 650.  So one warp fences
// while others add, every word has a thread of its own to wait for it, and the additions are
// spread over the quarters, a quantity to a warp.  A butterfly in every warp and one warp
// walking through flags and values took 12,000 to 29,000 clocks a sum; this, with the wait for the
// slowest block, 5,500 on 5x5 nodes, 7,800 at 161x81 and 10,900 at 2049x1025 (block 0's clocks).
struct alignas(16) SumWord {
    double v;
    unsigned long long seq;            // the sum the value belongs to; 0: none
};
constexpr int SUM_SPIN_LIMIT = 1 << 22;    // polls of about a third of a microsecond; then the launch gives up
constexpr int SUM_WORDS = 2 * 3 * MAX_SMS; // both sets, three quantities

__device__ __forceinline__ void sum_publish(SumWord *w, double v, unsigned long long seq) {
    asm volatile("{\n .reg .b128 t;\n mov.b128 t, {%1, %2};\n st.relaxed.gpu.global.b128 [%0], t;\n}"
                 ::"l"(w), "l"(__double_as_longlong(v)), "l"(seq) : "memory");
}
// acquire: what the publishing block wrote before can be read after
__device__ __forceinline__ void sum_read(const SumWord *w, double &v, unsigned long long &seq) {
    long long b;
    asm volatile("{\n .reg .b128 t;\n ld.acquire.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
                 : "=l"(b), "=l"(seq) : "l"(w) : "memory");
    v = __longlong_as_double(b);
}

// the totals over all blocks of Q <= 3 values of every thread (nact: this block's warps that have
// something to add), in a fixed order, left in tot (shared memory) for all threads; false: a
// block's sums did not arrive.  At least 16 warps.
struct SumShared {
    double sm[3][1024], part[3][4][32], all[3][MAX_SMS];
};
template <int Q>
__device__ __forceinline__ bool grid_totals(const double (&v)[Q], int nact, SumWord *words, unsigned long long seq,
                                            SumShared &S, double (&tot)[3]) {
    auto &sm = S.sm;
    auto &part = S.part;
    auto &all = S.all;
    const int t = threadIdx.x, w = t >> 5, l = t & 31, G = gridDim.x;
    SumWord *set = words + (seq & 1) * 3 * MAX_SMS;
    if (w < nact) {
#pragma unroll
        for (int q = 0; q < Q; ++q) sm[q][t] = v[q];
    }
    __syncthreads();                       // every thread's writes are done
    // the block's sums: warp 4 q + k the rows k, k + 4, ... of quantity q, then warp 4 q their four sums
    const int q = w >> 2, k = w & 3;
    if (q < Q) {
        double s = 0.0;
        for (int i = k; i < nact; i += 4) s += sm[q][i * 32 + l];
        part[q][k][l] = s;
        asm volatile("bar.sync %0, 128;" ::"r"(1 + q) : "memory");
        if (k == 0) {
            s = (part[q][0][l] + part[q][1][l]) + (part[q][2][l] + part[q][3][l]);
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (l == 0) tot[q] = s;
        }
    } else if (w == 15 && l == 0) {
        __threadfence();                   // the block's writes come before its sums
    }
    __syncthreads();
    if (t == 15 * 32) {
#pragma unroll
        for (int i = 0; i < Q; ++i) sum_publish(set + i * MAX_SMS + blockIdx.x, tot[i], seq);
    }
    bool ok = true;
    for (int i = t; i < Q * G; i += blockDim.x) {
        const int iq = i / G, b = i - iq * G;
        double x;
        unsigned long long got;
        int spins = 0;
        for (;;) {
            sum_read(set + iq * MAX_SMS + b, x, got);
            if (got == seq) break;
            if (++spins > SUM_SPIN_LIMIT) {
                ok = false;
                break;
            }
        }
        all[iq][b] = x;
    }
    ok = __syncthreads_and(ok);
    if (k == 0 && q < Q) {
        double s = 0.0;
        for (int b = l; b < G; b += 32) s += all[q][b];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (l == 0) tot[q] = s;
    }
    __syncthreads();
    return ok;
}

// the same without that: for a block's other words, when one of them is read by sum_read
__device__ __forceinline__ void sum_read_relaxed(const SumWord *w, double &v, unsigned long long &seq) {
    long long b;
    asm volatile("{\n .reg .b128 t;\n ld.relaxed.gpu.global.b128 t, [%2];\n mov.b128 {%0, %1}, t;\n}"
                 : "=l"(b), "=l"(seq) : "l"(w) : "memory");
    v = __longlong_as_double(b);
}

// The same totals, to the bit, by smaller blocks: a block of FEW_WARPS warps stands for nv (1, 2 or 4)
// of the G blocks above, p, p + gridDim.x, ... of them for block p.  Each of the G keeps its words and
// the order of its sums; the words from nwords on, whose blocks have nothing to add, are left out
// (nwords at least gridDim.x, since a block that publishes nothing would not be waited for).
// S.sm holds the values of the warps: row r of the k-th block at r nv + k, `rows` rows.
constexpr int FEW_WARPS = 8;
template <int ROWS>
struct SumSharedFew {
    double sm[3][ROWS * 32], half[3][32], part[3 * 4], all[3][MAX_SMS];
};
static_assert(MAX_SMS <= 32 * FEW_WARPS, "the words of a quantity have a thread each");
template <int Q, int ROWS>
__device__ __forceinline__ bool grid_totals_few(int nv, int rows, int nwords, SumWord *words, unsigned long long seq,
                                                SumSharedFew<ROWS> &S, double (&tot)[3]) {
    const int t = threadIdx.x, w = t >> 5, l = t & 31;
    SumWord *set = words + (seq & 1) * 3 * MAX_SMS;
    auto lanes_sum = [](double s) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        return s;
    };
    __syncthreads();                       // every thread's writes are done
    if (w == FEW_WARPS - 1) {
        if (l == 0) __threadfence();       // the block's writes come before its sums
    } else if (nv == 1) {                  // two warps a quantity: rows 4 i and 4 i + 1, 4 i + 2 and 4 i + 3
        const int q = w >> 1, k = 2 * (w & 1);
        if (q < Q) {
            double a = 0.0, b = 0.0;
            for (int r = k; r < rows; r += 4) {
                a += S.sm[q][r * 32 + l];
                if (r + 1 < rows) b += S.sm[q][(r + 1) * 32 + l];
            }
            if (k) S.half[q][l] = a + b;
            asm volatile("bar.sync %0, 64;" ::"r"(1 + q) : "memory");
            if (!k) {
                const double s = lanes_sum((a + b) + S.half[q][l]);
                if (l == 0) S.part[q] = s;
            }
        }
    } else {
        for (int j = w; j < Q * nv; j += FEW_WARPS - 1) {
            const int q = j / nv, k = j - q * nv;
            double p[4] = {0.0, 0.0, 0.0, 0.0};
#pragma unroll
            for (int r = 0; r < 4; ++r)
                if (r < rows) p[r] += S.sm[q][(r * nv + k) * 32 + l];
            const double s = lanes_sum((p[0] + p[1]) + (p[2] + p[3]));
            if (l == 0) S.part[j] = s;
        }
    }
    __syncthreads();
    if (t == (FEW_WARPS - 1) * 32) {
        for (int j = 0; j < Q * nv; ++j) {
            const int q = j / nv, b = blockIdx.x + (j - q * nv) * gridDim.x;
            if (b < nwords) sum_publish(set + q * MAX_SMS + b, S.part[j], seq);
        }
    }
    // The last quantity's words by one thread each, with acquire; the others' (at most two a thread) before
    // and without, so that a thread waits one round trip to L2 whatever its words
    const int N = FEW_WARPS * 32, m = (Q - 1) * nwords;
    bool ok = true;
    double x[2];
    unsigned long long got[2];
    auto word = [&](int i) { return set + i / nwords * MAX_SMS + i % nwords; };
#pragma unroll
    for (int j = 0; j < 2; ++j)
        if (N - 1 - t + j * N < m) sum_read_relaxed(word(N - 1 - t + j * N), x[j], got[j]);
    if (t < nwords) {
        double y;
        unsigned long long g;
        int spins = 0;
        for (;;) {
            sum_read(set + (Q - 1) * MAX_SMS + t, y, g);
            if (g == seq) break;
            if (++spins > SUM_SPIN_LIMIT) {
                ok = false;
                break;
            }
        }
        S.all[Q - 1][t] = y;
    }
#pragma unroll
    for (int j = 0; j < 2; ++j) {
        const int i = N - 1 - t + j * N;
        if (i >= m) break;
        for (int spins = 0; got[j] != seq; sum_read_relaxed(word(i), x[j], got[j]))
            if (++spins > SUM_SPIN_LIMIT) {
                ok = false;
                break;
            }
        S.all[i / nwords][i % nwords] = x[j];
    }
    ok = __syncthreads_and(ok);
    if (w < Q) {
        double s = 0.0;
        for (int b = l; b < nwords; b += 32) s += S.all[w][b];
        s = lanes_sum(s);
        if (l == 0) tot[w] = s;
    }
    __syncthreads();
    return ok;
}

}  // namespace bella
