// bk_engine.cuh -- the arithmetic "engines" of the operator kernels.
//
// Every kernel is written once over an engine that fixes
//   S  the storage type in HBM (double or float),
//   V  the working type in shared memory and registers,
//   C  the type of the 1-D matrix coefficients (kernel parameters),
//   A  the accumulator of a contraction,
// and the operations on them.  Engines:
//   EngDfma   FP64 storage, native FP64 FMA (1/64 of the FP32 rate on GB300);
//   EngFF     FP64 storage, float-float arithmetic on the FP32 pipes;
//   EngF32    FP32 storage and FMA: the reference drivers' T = float;
//   EngMixed  FP32 storage and FMA, with the final sum of the three
//             directional terms of BK3/BK5 compensated (TwoSum).
#pragma once

#include "bk_ff.cuh"

namespace bkg {

// The even and the odd half of a line's contraction (EOMat, EORMat) run side
// by side, one per lane: a coefficient pair C2 (even lane, odd lane), a value
// pair V2 and an accumulator pair A2 per engine.  The FP32-pipe engines use
// packed operations (two lanes per instruction, bk_ff.cuh), the DFMA engine
// two doubles.
template <class C>
struct CoefPair;
template <>
struct CoefPair<double> {
    double x, y;
    void set(double a, double b)
    {
        x = a;
        y = b;
    }
};
template <>
struct CoefPair<float> {
    f2 v;
    void set(float a, float b) { v = f2_make(a, b); }
};
template <>
struct CoefPair<ff> : ffcp {
    void set(ff a, ff b)
    {
        x = a;
        y = b;
    }
};

struct EngDfma {
    using S = double;
    using V = double;
    using C = double;
    using A = double;
    static constexpr int kId = BK_ENGINE_DFMA;
    __device__ static __forceinline__ V load(S x) { return x; }
    template <int N>
    __device__ static __forceinline__ void load_n(const S (&x)[N], V (&y)[N])
    {
#pragma unroll
        for (int i = 0; i < N; ++i) y[i] = x[i];
    }
    __device__ static __forceinline__ S store(V x) { return x; }
    __device__ static __forceinline__ S store(V x, bool) { return x; }
    __device__ static __forceinline__ A zero() { return 0.0; }
    // an accumulator started with a first product / value (no add to zero)
    __device__ static __forceinline__ A first(C c, V x) { return c * x; }
    __device__ static __forceinline__ A vfirst(V a, V x) { return a * x; }
    __device__ static __forceinline__ A from(V x) { return x; }
    __device__ static __forceinline__ void madd(A& acc, C c, V x) { acc = fma(c, x, acc); }
    __device__ static __forceinline__ void vmadd(A& acc, V a, V x) { acc = fma(a, x, acc); }
    __device__ static __forceinline__ void add(A& acc, V x) { acc += x; }
    __device__ static __forceinline__ V result(A acc) { return acc; }
    __device__ static __forceinline__ V loose(A acc) { return acc; }
    __device__ static __forceinline__ V mul(V a, V b) { return a * b; }
    struct V2 {
        V x, y;
    };
    using A2 = V2;
    // (a + b, a - b): the even and odd combinations of two line values
    __device__ static __forceinline__ V2 even_odd(V a, V b) { return V2{a + b, a - b}; }
    __device__ static __forceinline__ V even(const V2& v) { return v.x; }
    __device__ static __forceinline__ V odd(const V2& v) { return v.y; }
    __device__ static __forceinline__ A2 first2(const CoefPair<C>& c, const V2& v) { return A2{c.x * v.x, c.y * v.y}; }
    __device__ static __forceinline__ void madd2(A2& acc, const CoefPair<C>& c, const V2& v)
    {
        acc.x = fma(c.x, v.x, acc.x);
        acc.y = fma(c.y, v.y, acc.y);
    }
    // the even lane alone
    __device__ static __forceinline__ void madd_even(A2& acc, C c, V x) { acc.x = fma(c, x, acc.x); }
    // s = even + odd; d = odd - even (SIGN < 0) or even - odd (SIGN > 0)
    template <int SIGN, bool LOOSE>
    __device__ static __forceinline__ void sum_diff(const A2& a, V& s, V& d)
    {
        s = a.x + a.y;
        d = SIGN > 0 ? a.x - a.y : a.y - a.x;
    }
    static C coef(double d) { return d; }
};

struct EngFF {
    using S = double;
    using V = ff;
    using C = ff;
    using A = ffacc;
    static constexpr int kId = BK_ENGINE_FF;
    __device__ static __forceinline__ V load(S x) { return split(x); }
    // a value split ahead of time (bk_g_to_ff): no work
    __device__ static __forceinline__ V load(ff2 x) { return ff{x.hi, x.lo}; }
    template <int N>
    __device__ static __forceinline__ void load_n(const S (&x)[N], V (&y)[N])
    {
        split_n(x, y);
    }
    template <int N>
    __device__ static __forceinline__ void load_n(const ff2 (&x)[N], V (&y)[N])
    {
#pragma unroll
        for (int i = 0; i < N; ++i) y[i] = load(x[i]);
    }
    __device__ static __forceinline__ S store(V x) { return join(x); }
    // fp64: on the FP64 pipe
    __device__ static __forceinline__ S store(V x, bool fp64) { return fp64 ? join_fp64(x) : join(x); }
    __device__ static __forceinline__ A zero() { return acc_zero(); }
    // the first product needs no TwoSum into an empty accumulator
    __device__ static __forceinline__ A first(C c, V x) { return acc_first(c, x); }
    __device__ static __forceinline__ A vfirst(V a, V x) { return acc_first(a, x); }
    __device__ static __forceinline__ A from(V x) { return ffacc{x.hi, x.lo}; }
    __device__ static __forceinline__ void madd(A& acc, C c, V x) { acc_madd(acc, c, x); }
    __device__ static __forceinline__ void vmadd(A& acc, V a, V x) { acc_madd(acc, a, x); }
    __device__ static __forceinline__ void add(A& acc, V x) { acc_add(acc, x); }
    __device__ static __forceinline__ V result(A acc) { return acc_result(acc); }
    // for values that are only summed or stored next: not renormalised
    __device__ static __forceinline__ V loose(A acc) { return acc_loose(acc); }
    __device__ static __forceinline__ V mul(V a, V b) { return ff_mul(a, b); }
    using V2 = ffp;
    using A2 = ffaccp;
    // operands of multiply-adds only: not renormalised
    __device__ static __forceinline__ V2 even_odd(V a, V b)
    {
        return ffp{ff_add_loose(a, b), ff_add_loose(a, ff{-b.hi, -b.lo})};
    }
    __device__ static __forceinline__ V even(const V2& v) { return v.x; }
    __device__ static __forceinline__ V odd(const V2& v) { return v.y; }
    __device__ static __forceinline__ A2 first2(const CoefPair<C>& c, const V2& v) { return acc_first2(c, v); }
    __device__ static __forceinline__ void madd2(A2& acc, const CoefPair<C>& c, const V2& v) { acc_madd2(acc, c, v); }
    __device__ static __forceinline__ void madd_even(A2& acc, C c, V x)
    {
        ffacc a{f2_x(acc.s), f2_x(acc.c)};
        acc_madd(a, c, x);
        acc = A2{f2_make(a.s, f2_y(acc.s)), f2_make(a.c, f2_y(acc.c))};
    }
    // LOOSE: unevaluated pairs, for outputs that are only summed next
    template <int SIGN, bool LOOSE>
    __device__ static __forceinline__ void sum_diff(const A2& ab, V& s, V& d)
    {
        const ffacc a{f2_x(ab.s), f2_x(ab.c)}, b{f2_y(ab.s), f2_y(ab.c)};
        if constexpr (LOOSE) {
            if constexpr (SIGN > 0) acc_sum_diff_loose(b, a, s, d);
            else acc_sum_diff_loose(a, b, s, d);
        } else {
            if constexpr (SIGN > 0) acc_sum_diff(b, a, s, d);
            else acc_sum_diff(a, b, s, d);
        }
    }
    static C coef(double d)
    {
        C c;
        c.hi = static_cast<float>(d);
        c.lo = static_cast<float>(d - static_cast<double>(c.hi));
        return c;
    }
};

struct EngF32 {
    using S = float;
    using V = float;
    using C = float;
    using A = float;
    static constexpr int kId = 100;
    __device__ static __forceinline__ V load(S x) { return x; }
    template <int N>
    __device__ static __forceinline__ void load_n(const S (&x)[N], V (&y)[N])
    {
#pragma unroll
        for (int i = 0; i < N; ++i) y[i] = x[i];
    }
    __device__ static __forceinline__ S store(V x) { return x; }
    __device__ static __forceinline__ S store(V x, bool) { return x; }
    __device__ static __forceinline__ A zero() { return 0.0f; }
    __device__ static __forceinline__ A first(C c, V x) { return c * x; }
    __device__ static __forceinline__ A vfirst(V a, V x) { return a * x; }
    __device__ static __forceinline__ A from(V x) { return x; }
    __device__ static __forceinline__ void madd(A& acc, C c, V x) { acc = fmaf(c, x, acc); }
    __device__ static __forceinline__ void vmadd(A& acc, V a, V x) { acc = fmaf(a, x, acc); }
    __device__ static __forceinline__ void add(A& acc, V x) { acc += x; }
    __device__ static __forceinline__ V result(A acc) { return acc; }
    __device__ static __forceinline__ V loose(A acc) { return acc; }
    __device__ static __forceinline__ V mul(V a, V b) { return a * b; }
    using V2 = f2;
    using A2 = f2;
    __device__ static __forceinline__ V2 even_odd(V a, V b) { return f2_make(a + b, a - b); }
    __device__ static __forceinline__ V even(V2 v) { return f2_x(v); }
    __device__ static __forceinline__ V odd(V2 v) { return f2_y(v); }
    __device__ static __forceinline__ A2 first2(const CoefPair<C>& c, V2 v) { return f2_mul(c.v, v); }
    __device__ static __forceinline__ void madd2(A2& acc, const CoefPair<C>& c, V2 v) { acc = f2_fma(c.v, v, acc); }
    __device__ static __forceinline__ void madd_even(A2& acc, C c, V x)
    {
        acc = f2_make(fmaf(c, x, f2_x(acc)), f2_y(acc));
    }
    template <int SIGN, bool LOOSE>
    __device__ static __forceinline__ void sum_diff(A2 a, V& s, V& d)
    {
        s = f2_x(a) + f2_y(a);
        d = SIGN > 0 ? f2_x(a) - f2_y(a) : f2_y(a) - f2_x(a);
    }
    static C coef(double d) { return static_cast<float>(d); }
};

// Plain FP32 everywhere except the final combination of the three directional
// terms, which is summed with TwoSum and rounded once.
struct EngMixed : EngF32 {
    static constexpr int kId = 101;
    __device__ static __forceinline__ float sum3(float a, float b, float c)
    {
        float s, e, s2, e2;
        two_sum(a, b, s, e);
        two_sum(s, c, s2, e2);
        return __fadd_rn(s2, __fadd_rn(e, e2));
    }
};

template <class Eng>
struct HasSum3 {
    static constexpr bool value = false;
};
template <>
struct HasSum3<EngMixed> {
    static constexpr bool value = true;
};

}  // namespace bkg
