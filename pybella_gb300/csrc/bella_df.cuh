// bella_df.cuh -- double-float ("FP32 pair") arithmetic for the Krylov path.
//
// GB300 executes FP64 at 1/64 of its FP32 rate (measured 1.01 vs 64.2
// TFLOP/s), which makes the FP64 stencil FP64-pipe bound at ~14 % of HBM
// bandwidth.  A value is kept as hi + lo with |lo| <= ulp(hi)/2 (about 48
// significant bits, ~1e-14 relative) and operated on with error-free
// transformations on the FP32 pipe:
//   two-sum (Knuth), fast-two-sum (Dekker), two-product via fmaf,
// following Dekker (1971) / Knuth TAOCP vol. 2 and the double-double
// algorithms of Hida, Li & Bailey (2001).  Every operation uses the _rn
// intrinsics so the compiler cannot contract or reassociate them.
#pragma once
#include <cuda_runtime.h>

namespace bella {

struct __align__(8) dfloat {
    float hi, lo;
    __host__ __device__ __forceinline__ dfloat() {}
    __host__ __device__ __forceinline__ dfloat(float h, float l) : hi(h), lo(l) {}
    __device__ __forceinline__ dfloat(int v) : hi((float)v), lo(0.f) {}
    __device__ __forceinline__ dfloat(double d) {
        hi = __double2float_rn(d);
        lo = __double2float_rn(d - (double)hi);
    }
    __device__ __forceinline__ double to_double() const { return (double)hi + (double)lo; }
};

// s + e == a + b exactly
__device__ __forceinline__ void two_sum(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    const float bb = __fsub_rn(s, a);
    e = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
}

// requires |a| >= |b| (or a == 0)
__device__ __forceinline__ void fast_two_sum(float a, float b, float &s, float &e) {
    s = __fadd_rn(a, b);
    e = __fsub_rn(b, __fsub_rn(s, a));
}

// accurate double-float sum (relative error ~2^-47 even under cancellation)
__device__ __forceinline__ dfloat df_add(dfloat a, dfloat b) {
    float s, e, t, f;
    two_sum(a.hi, b.hi, s, e);
    two_sum(a.lo, b.lo, t, f);
    e = __fadd_rn(e, t);
    fast_two_sum(s, e, s, e);
    e = __fadd_rn(e, f);
    fast_two_sum(s, e, s, e);
    return dfloat(s, e);
}

__device__ __forceinline__ dfloat df_neg(dfloat a) { return dfloat(-a.hi, -a.lo); }

__device__ __forceinline__ dfloat df_mul(dfloat a, dfloat b) {
    const float p = __fmul_rn(a.hi, b.hi);
    float e = __fmaf_rn(a.hi, b.hi, -p);
    e = __fmaf_rn(a.hi, b.lo, e);
    e = __fmaf_rn(a.lo, b.hi, e);
    float s;
    fast_two_sum(p, e, s, e);
    return dfloat(s, e);
}

__device__ __forceinline__ dfloat operator+(dfloat a, dfloat b) { return df_add(a, b); }
__device__ __forceinline__ dfloat operator-(dfloat a, dfloat b) { return df_add(a, df_neg(b)); }
__device__ __forceinline__ dfloat operator*(dfloat a, dfloat b) { return df_mul(a, b); }
__device__ __forceinline__ dfloat &operator+=(dfloat &a, dfloat b) { a = df_add(a, b); return a; }

// Inner-product accumulator: each product a*b of two double-floats is formed
// to ~2^-48 relative (exact hi*hi via fmaf plus the cross terms) and summed
// into a compensated FP32 pair; converted to FP64 once per thread.
struct DFAcc {
    float hi, lo;
    __device__ __forceinline__ void zero() { hi = 0.f; lo = 0.f; }
    __device__ __forceinline__ void add_prod(dfloat a, dfloat b) {
        const float p = __fmul_rn(a.hi, b.hi);
        float e = __fmaf_rn(a.hi, b.hi, -p);
        e = __fmaf_rn(a.hi, b.lo, e);
        e = __fmaf_rn(a.lo, b.hi, e);
        float s, err;
        two_sum(hi, p, s, err);
        hi = s;
        lo = __fadd_rn(lo, __fadd_rn(err, e));
    }
    __device__ __forceinline__ double value() const { return (double)hi + (double)lo; }
};

// ---- two double-floats at once on Blackwell's packed FP32 instructions -----------
// (add / sub / mul / fma.rn.f32x2: two FP32 operations an instruction, each rounded as the scalar
// one).  The operator's double-float arithmetic is issue-bound: 254 FP32 instructions a node of the
// 2D p-direction stencil and as many again around them; in pairs, half.  Every operation is
// the scalar one's, value for value.
typedef unsigned long long f32x2;              // (low word: first value, high word: second)

__device__ __forceinline__ f32x2 x2_pack(float a, float b) {
    f32x2 r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ void x2_unpack(f32x2 v, float &a, float &b) {
    asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(v));
}
__device__ __forceinline__ f32x2 x2_add(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 x2_sub(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("sub.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 x2_mul(f32x2 a, f32x2 b) {
    f32x2 r;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r) : "l"(a), "l"(b));
    return r;
}
__device__ __forceinline__ f32x2 x2_fma(f32x2 a, f32x2 b, f32x2 c) {
    f32x2 r;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r) : "l"(a), "l"(b), "l"(c));
    return r;
}
__device__ __forceinline__ f32x2 x2_neg(f32x2 a) { return a ^ 0x8000000080000000ull; }

struct dfloat2 {
    f32x2 hi, lo;
    __device__ __forceinline__ dfloat2() {}
    __device__ __forceinline__ dfloat2(f32x2 h, f32x2 l) : hi(h), lo(l) {}
    __device__ __forceinline__ dfloat2(dfloat a, dfloat b) : hi(x2_pack(a.hi, b.hi)), lo(x2_pack(a.lo, b.lo)) {}
    __device__ __forceinline__ void split(dfloat &a, dfloat &b) const {
        x2_unpack(hi, a.hi, b.hi);
        x2_unpack(lo, a.lo, b.lo);
    }
};

// the tail of a sum: s + e with the low words' sum t + f folded in
__device__ __forceinline__ dfloat2 x2_renorm(f32x2 s, f32x2 e, f32x2 t, f32x2 f) {
    e = x2_add(e, t);
    f32x2 q = x2_add(s, e);
    e = x2_add(x2_sub(e, x2_sub(q, s)), f);
    s = x2_add(q, e);
    return dfloat2(s, x2_sub(e, x2_sub(s, q)));
}
__device__ __forceinline__ void x2_two_sum(f32x2 a, f32x2 b, f32x2 &s, f32x2 &e) {
    s = x2_add(a, b);
    const f32x2 bb = x2_sub(s, a);
    e = x2_add(x2_sub(a, x2_sub(s, bb)), x2_sub(b, bb));
}
__device__ __forceinline__ void x2_two_diff(f32x2 a, f32x2 b, f32x2 &s, f32x2 &e) {
    s = x2_sub(a, b);
    const f32x2 bb = x2_sub(s, a);
    e = x2_sub(x2_sub(a, x2_sub(s, bb)), x2_add(b, bb));
}
__device__ __forceinline__ dfloat2 operator+(dfloat2 a, dfloat2 b) {
    f32x2 s, e, t, f;
    x2_two_sum(a.hi, b.hi, s, e);
    x2_two_sum(a.lo, b.lo, t, f);
    return x2_renorm(s, e, t, f);
}
__device__ __forceinline__ dfloat2 operator-(dfloat2 a, dfloat2 b) {
    f32x2 s, e, t, f;
    x2_two_diff(a.hi, b.hi, s, e);
    x2_two_diff(a.lo, b.lo, t, f);
    return x2_renorm(s, e, t, f);
}
__device__ __forceinline__ dfloat2 operator*(dfloat2 a, dfloat2 b) {
    const f32x2 p = x2_mul(a.hi, b.hi);
    f32x2 e = x2_fma(a.hi, b.hi, x2_neg(p));
    e = x2_fma(a.hi, b.lo, e);
    e = x2_fma(a.lo, b.hi, e);
    const f32x2 s = x2_add(p, e);
    return dfloat2(s, x2_sub(e, x2_sub(s, p)));
}

// DFAcc of two sequences of products
struct DFAcc2 {
    f32x2 hi, lo;
    __device__ __forceinline__ void zero() { hi = 0ull; lo = 0ull; }
    __device__ __forceinline__ void add_prod(dfloat2 a, dfloat2 b) {
        const f32x2 p = x2_mul(a.hi, b.hi);
        f32x2 e = x2_fma(a.hi, b.hi, x2_neg(p));
        e = x2_fma(a.hi, b.lo, e);
        e = x2_fma(a.lo, b.hi, e);
        f32x2 s, err;
        x2_two_sum(hi, p, s, err);
        hi = s;
        lo = x2_add(lo, x2_add(err, e));
    }
    __device__ __forceinline__ double value() const {
        float h0, h1, l0, l1;
        x2_unpack(hi, h0, h1);
        x2_unpack(lo, l0, l1);
        return ((double)h0 + (double)l0) + ((double)h1 + (double)l1);
    }
};

}  // namespace bella
