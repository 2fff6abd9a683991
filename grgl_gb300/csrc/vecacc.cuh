// Per-lane accumulators for the VW columns a lane owns in the sweep.
//
// The generic VecAcc keeps one scalar accumulator per column.  The compensated float32 and the
// float-pair float64 operators keep their state as float2 pairs of adjacent columns (structure
// of arrays), so every addition is a packed FP32x2 instruction (FADD2, or FFMA2 with a -1
// multiplier for an exact subtraction) on register pairs that need no repacking.
#pragma once
#include "ops.cuh"

namespace grgx {

// ---- packed float2 arithmetic (Blackwell FADD2 / FFMA2) --------------------------------------
// Each operation rounds exactly like the scalar __fadd_rn / __fsub_rn of its component.
__device__ __forceinline__ float2 add2(float2 a, float2 b) { return __fadd2_rn(a, b); }
__device__ __forceinline__ float2 sub2(float2 a, float2 b) { return __ffma2_rn(b, make_float2(-1.0f, -1.0f), a); }
__device__ __forceinline__ float2 shfl_xor2(float2 a, int m) {
    return make_float2(__shfl_xor_sync(FULL_MASK, a.x, m), __shfl_xor_sync(FULL_MASK, a.y, m));
}
__device__ __forceinline__ float2 shfl_up2(float2 a, int d) {
    return make_float2(__shfl_up_sync(FULL_MASK, a.x, d), __shfl_up_sync(FULL_MASK, a.y, d));
}
__device__ __forceinline__ float lane_of(float2 a, int i) { return (i & 1) ? a.y : a.x; }

// TwoSum on pairs: s = a + b rounded, e = exact error.
__device__ __forceinline__ void two_sum2(float2 a, float2 b, float2& s, float2& e) {
    s = add2(a, b);
    const float2 bb = sub2(s, a);
    e = add2(sub2(a, sub2(s, bb)), sub2(b, bb));
}

// One Op::A accumulator per column (the generic accumulator; also used directly where a kernel
// wants the scalar form of a type VecAcc specialises).
template <class Op, int VW> struct ScalarAcc {
    using S = typename Op::S;
    using A = typename Op::A;
    A a[VW];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < VW; i++) a[i] = Op::zero();
    }
    __device__ __forceinline__ void add(const S* v) {
#pragma unroll
        for (int i = 0; i < VW; i++) Op::add(a[i], v[i]);
    }
    // N consecutive edges of one row (the sweep's boundary-free steps).
    template <int N> __device__ __forceinline__ void add_block(const S (*v)[VW]) {
#pragma unroll
        for (int u = 0; u < N; u++) add(v[u]);
    }
    // Four pattern rows of the pair form, each the sum of two edges' rows.
    __device__ __forceinline__ void add_pairs(const S (*v)[VW]) { add_block<4>(v); }
    __device__ __forceinline__ void merge(const ScalarAcc& o) {
#pragma unroll
        for (int i = 0; i < VW; i++) Op::merge(a[i], o.a[i]);
    }
    __device__ __forceinline__ ScalarAcc shfl_xor(int m) const {
        ScalarAcc r;
#pragma unroll
        for (int i = 0; i < VW; i++) r.a[i] = Op::shfl_xor(a[i], m);
        return r;
    }
    __device__ __forceinline__ ScalarAcc shfl_up(int d) const {
        ScalarAcc r;
#pragma unroll
        for (int i = 0; i < VW; i++) r.a[i] = Op::shfl_up(a[i], d);
        return r;
    }
    __device__ __forceinline__ A get(int i) const { return a[i]; }
    __device__ __forceinline__ void add_partial(int i, const A& x) { Op::merge(a[i], x); }
    __device__ __forceinline__ void settle() {}
    __device__ __forceinline__ void flush() {}
};

template <class Op, int VW> struct VecAcc : ScalarAcc<Op, VW> {
    __device__ __forceinline__ VecAcc() = default;
    __device__ __forceinline__ VecAcc(const ScalarAcc<Op, VW>& s) : ScalarAcc<Op, VW>(s) {}
    __device__ __forceinline__ VecAcc shfl_xor(int m) const { return VecAcc(ScalarAcc<Op, VW>::shfl_xor(m)); }
    __device__ __forceinline__ VecAcc shfl_up(int d) const { return VecAcc(ScalarAcc<Op, VW>::shfl_up(d)); }
};

// Compensated float32, one column (K = 1): two independent compensated partial sums in the .x
// and .y halves of float2 registers, so a boundary-free step adds its edges two at a time with
// packed TwoSums (FADD2); single adds go to .x.  get() merges the halves (one more TwoSum), and
// merges, shuffles and partials work half by half.  Per node the error stays that of a
// compensated sum: each half's running error is carried exactly until the final merge.
template <> struct VecAcc<AddF32C, 1> {
    using S = float;
    using A = F32Pair;
    float2 hi, lo;
    __device__ __forceinline__ void zero() { hi = lo = make_float2(0.0f, 0.0f); }
    __device__ __forceinline__ void add(const float* v) {
        A x{hi.x, lo.x};
        AddF32C::add(x, v[0]);
        hi.x = x.hi;
        lo.x = x.lo;
    }
    template <int N> __device__ __forceinline__ void add_block(const float (*v)[1]) {
#pragma unroll
        for (int u = 0; u + 1 < N; u += 2) {
            float2 sum, err;
            two_sum2(hi, make_float2(v[u][0], v[u + 1][0]), sum, err);
            hi = sum;
            lo = add2(lo, err);
        }
        if (N & 1) add(v[N - 1]);
    }
    // Four pattern rows of the pair form with their errors.
    __device__ __forceinline__ void add_pairs(const F32Pair (*v)[1]) {
#pragma unroll
        for (int u = 0; u < 4; u += 2) {
            float2 sum, err;
            two_sum2(hi, make_float2(v[u][0].hi, v[u + 1][0].hi), sum, err);
            hi = sum;
            lo = add2(lo, add2(err, make_float2(v[u][0].lo, v[u + 1][0].lo)));
        }
    }
    __device__ __forceinline__ void merge(const VecAcc& o) {
        float2 sum, err;
        two_sum2(hi, o.hi, sum, err);
        hi = sum;
        lo = add2(lo, add2(o.lo, err));
    }
    __device__ __forceinline__ VecAcc shfl_xor(int m) const {
        VecAcc r;
        r.hi = shfl_xor2(hi, m);
        r.lo = shfl_xor2(lo, m);
        return r;
    }
    __device__ __forceinline__ VecAcc shfl_up(int d) const {
        VecAcc r;
        r.hi = shfl_up2(hi, d);
        r.lo = shfl_up2(lo, d);
        return r;
    }
    __device__ __forceinline__ A get(int) const {
        A x{hi.x, lo.x};
        AddF32C::merge(x, A{hi.y, lo.y});
        return x;
    }
    __device__ __forceinline__ void add_partial(int, const A& p) {
        A x{hi.x, lo.x};
        AddF32C::merge(x, p);
        hi.x = x.hi;
        lo.x = x.lo;
    }
    __device__ __forceinline__ void settle() {}
    __device__ __forceinline__ void flush() {}
};

// float64 as float pairs, one column (K = 1): scalar state with periodic renormalisation.
template <> struct VecAcc<AddF64S, 1> {
    F64Run a[1];
    __device__ __forceinline__ void zero() { a[0] = AddF64S::zero(); }
    __device__ __forceinline__ void add(const DF* v) { AddF64S::add(a[0], v[0]); }
    template <int N> __device__ __forceinline__ void add_block(const DF (*v)[1]) {
#pragma unroll
        for (int u = 0; u < N; u++) {
            add(v[u]);
            if ((u & 3) == 3) settle();
        }
    }
    __device__ __forceinline__ void merge(const VecAcc& o) { AddF64S::merge(a[0], o.a[0]); }
    __device__ __forceinline__ VecAcc shfl_xor(int m) const { return {{AddF64S::shfl_xor(a[0], m)}}; }
    __device__ __forceinline__ VecAcc shfl_up(int d) const { return {{AddF64S::shfl_up(a[0], d)}}; }
    __device__ __forceinline__ F64Run get(int) const { return a[0]; }
    __device__ __forceinline__ void add_partial(int, const F64Run& x) { AddF64S::merge(a[0], x); }
    __device__ __forceinline__ void settle() { AddF64S::settle(a[0]); }
    __device__ __forceinline__ void flush() { AddF64S::flush(a[0]); }
};

// In boundary-free steps the edges of a row are added in plain float32 four at a time, as a
// two-level tree, before one TwoSum takes the quad into the compensated (hi, lo) pair.  A node's
// error then stays within 2u * sum|x| (the tree roundings) + u * |value| (its final rounding),
// u = 2^-24, for a quarter of the TwoSums of one per edge; steps with a row boundary keep one
// TwoSum per edge.
constexpr int kF32PreSum = 4;
// No pre-sum: a FastTwoSum (Dekker, Numer. Math. 18, 1971) of running sum and addend per edge, four
// operations as one of two edges behind a pre-sum has.  Its error term is exact where the sum is not the
// smaller of the two -- nearly always once a few edges are in it -- and otherwise off by at most the rounding
// that a plain addition has.
constexpr int kF32Ordered = 0;

// Compensated float32, columns in pairs; PRE edges are pre-summed in add_block.
template <int NP, int PRE = kF32PreSum> struct PackedF32C {
    float2 hi[NP], lo[NP];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int j = 0; j < NP; j++) hi[j] = lo[j] = make_float2(0.0f, 0.0f);
    }
    __device__ __forceinline__ void add_pair2(int j, float2 x) {
        float2 s, e;
        two_sum2(hi[j], x, s, e);
        lo[j] = add2(lo[j], e);
        hi[j] = s;
    }
    __device__ __forceinline__ void add(const float* v) {
#pragma unroll
        for (int j = 0; j < NP; j++) add_pair2(j, make_float2(v[2 * j], v[2 * j + 1]));
    }
    __device__ __forceinline__ void add_ordered(const float* v) {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            const float2 x = make_float2(v[2 * j], v[2 * j + 1]), s = add2(hi[j], x);
            lo[j] = add2(lo[j], sub2(x, sub2(s, hi[j])));
            hi[j] = s;
        }
    }
    template <int N> __device__ __forceinline__ void add_block(const float (*v)[2 * NP]) {
        if constexpr (PRE == kF32PreSum) {
            static_assert(N % PRE == 0 && PRE == 4, "block of whole pre-sums");
#pragma unroll
            for (int u = 0; u < N; u += PRE) {
#pragma unroll
                for (int j = 0; j < NP; j++) {
                    const float2 a = make_float2(v[u][2 * j], v[u][2 * j + 1]);
                    const float2 b = make_float2(v[u + 1][2 * j], v[u + 1][2 * j + 1]);
                    const float2 c = make_float2(v[u + 2][2 * j], v[u + 2][2 * j + 1]);
                    const float2 d = make_float2(v[u + 3][2 * j], v[u + 3][2 * j + 1]);
                    add_pair2(j, add2(add2(a, b), add2(c, d)));
                }
            }
        } else {
            static_assert(N % 2 == 0 && (PRE == 1 || PRE == 2 || PRE == kF32Ordered), "no other pre-sums");
#pragma unroll
            for (int u = 0; u < N; u++) {
                if constexpr (PRE == 1) {
                    add(v[u]);
                } else if constexpr (PRE == 2) {
#pragma unroll
                    for (int j = 0; u % 2 == 0 && j < NP; j++)
                        add_pair2(j, add2(make_float2(v[u][2 * j], v[u][2 * j + 1]), make_float2(v[u + 1][2 * j], v[u + 1][2 * j + 1])));
                } else {
                    add_ordered(v[u]);
                }
            }
        }
    }
    // Four pattern rows of the pair form, each the rounded sum of two edges.
    __device__ __forceinline__ void add_pairs(const float (*v)[2 * NP]) {
        static_assert(PRE == 1 || PRE == kF32Ordered, "a pattern row is a pre-sum already");
        add_block<4>(v);
    }
    __device__ __forceinline__ void merge(const PackedF32C& o) {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            float2 s, e;
            two_sum2(hi[j], o.hi[j], s, e);
            lo[j] = add2(lo[j], add2(o.lo[j], e));
            hi[j] = s;
        }
    }
    __device__ __forceinline__ PackedF32C shfl_xor(int m) const {
        PackedF32C r;
#pragma unroll
        for (int j = 0; j < NP; j++) {
            r.hi[j] = shfl_xor2(hi[j], m);
            r.lo[j] = shfl_xor2(lo[j], m);
        }
        return r;
    }
    __device__ __forceinline__ PackedF32C shfl_up(int d) const {
        PackedF32C r;
#pragma unroll
        for (int j = 0; j < NP; j++) {
            r.hi[j] = shfl_up2(hi[j], d);
            r.lo[j] = shfl_up2(lo[j], d);
        }
        return r;
    }
    __device__ __forceinline__ F32Pair get(int i) const { return {lane_of(hi[i >> 1], i), lane_of(lo[i >> 1], i)}; }
    __device__ __forceinline__ void add_partial(int i, const F32Pair& x) {
        F32Pair r = get(i);
        AddF32C::merge(r, x);
        if (i & 1) {
            hi[i >> 1].y = r.hi;
            lo[i >> 1].y = r.lo;
        } else {
            hi[i >> 1].x = r.hi;
            lo[i >> 1].x = r.lo;
        }
    }
    __device__ __forceinline__ void settle() {}
    __device__ __forceinline__ void flush() {}
};
template <> struct VecAcc<AddF32C, 2> : PackedF32C<1> {};
template <> struct VecAcc<AddF32C, 4> : PackedF32C<2> {};
template <> struct VecAcc<AddF32CX, 2> : PackedF32C<1, 1> {
    __device__ __forceinline__ void add_pairs(const F32Pair (*v)[2]) {
#pragma unroll
        for (int u = 0; u < 4; u++) {
            add_pair2(0, make_float2(v[u][0].hi, v[u][1].hi));
            lo[0] = add2(lo[0], make_float2(v[u][0].lo, v[u][1].lo));
        }
    }
};
template <int PRE> struct VecAcc<AddF32CPre<PRE>, 1> : VecAcc<AddF32C, 1> {};
template <int PRE> struct VecAcc<AddF32CPre<PRE>, 2> : PackedF32C<1, PRE> {};
template <int PRE> struct VecAcc<AddF32CPre<PRE>, 4> : PackedF32C<2, PRE> {};

// float64 as float pairs, columns in pairs: double run folds, float2 (hi, lo) state.
template <int NP> struct PackedF64S {
    double acc[2 * NP];
    float2 hi[NP], lo[NP];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            acc[2 * j] = acc[2 * j + 1] = 0.0;
            hi[j] = lo[j] = make_float2(0.0f, 0.0f);
        }
    }
    __device__ __forceinline__ void add(const DF* v) {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            const float2 xh = make_float2(v[2 * j].hi, v[2 * j + 1].hi);
            const float2 xl = make_float2(v[2 * j].lo, v[2 * j + 1].lo);
            float2 s, e;
            two_sum2(hi[j], xh, s, e);
            lo[j] = add2(lo[j], add2(e, xl));
            hi[j] = s;
        }
    }
    template <int N> __device__ __forceinline__ void add_block(const DF (*v)[2 * NP]) {
#pragma unroll
        for (int u = 0; u < N; u++) {
            add(v[u]);
            if ((u & 3) == 3) settle();
        }
    }
    __device__ __forceinline__ void settle() {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            const float2 h = add2(hi[j], lo[j]);
            lo[j] = sub2(lo[j], sub2(h, hi[j]));
            hi[j] = h;
        }
    }
    __device__ __forceinline__ F64Run get(int i) const {
        return {acc[i], lane_of(hi[i >> 1], i), lane_of(lo[i >> 1], i)};
    }
    __device__ __forceinline__ void set(int i, const F64Run& r) {
        acc[i] = r.acc;
        if (i & 1) {
            hi[i >> 1].y = r.hi;
            lo[i >> 1].y = r.lo;
        } else {
            hi[i >> 1].x = r.hi;
            lo[i >> 1].x = r.lo;
        }
    }
    __device__ __forceinline__ void flush() {
#pragma unroll
        for (int i = 0; i < 2 * NP; i++) {
            F64Run r = get(i);
            AddF64S::flush(r);
            set(i, r);
        }
    }
    __device__ __forceinline__ void add_partial(int i, const F64Run& x) {
        F64Run r = get(i);
        AddF64S::merge(r, x);
        set(i, r);
    }
    __device__ __forceinline__ void merge(const PackedF64S& o) {
#pragma unroll
        for (int i = 0; i < 2 * NP; i++) {
            F64Run r = get(i);
            AddF64S::merge(r, o.get(i));
            set(i, r);
        }
    }
    __device__ __forceinline__ PackedF64S shfl_xor(int m) const {
        PackedF64S r;
#pragma unroll
        for (int j = 0; j < NP; j++) {
            r.acc[2 * j] = __shfl_xor_sync(FULL_MASK, acc[2 * j], m);
            r.acc[2 * j + 1] = __shfl_xor_sync(FULL_MASK, acc[2 * j + 1], m);
            r.hi[j] = shfl_xor2(hi[j], m);
            r.lo[j] = shfl_xor2(lo[j], m);
        }
        return r;
    }
    __device__ __forceinline__ PackedF64S shfl_up(int d) const {
        PackedF64S r;
#pragma unroll
        for (int j = 0; j < NP; j++) {
            r.acc[2 * j] = __shfl_up_sync(FULL_MASK, acc[2 * j], d);
            r.acc[2 * j + 1] = __shfl_up_sync(FULL_MASK, acc[2 * j + 1], d);
            r.hi[j] = shfl_up2(hi[j], d);
            r.lo[j] = shfl_up2(lo[j], d);
        }
        return r;
    }
};
template <> struct VecAcc<AddF64S, 2> : PackedF64S<1> {};

// df_add on pairs of columns.
__device__ __forceinline__ void df_add2(float2& ahi, float2& alo, float2 bhi, float2 blo) {
    float2 s, e, t, f, g, h;
    two_sum2(ahi, bhi, s, e);
    two_sum2(alo, blo, t, f);
    two_sum2(e, t, g, h);
    ahi = add2(s, g);
    alo = add2(sub2(g, sub2(ahi, s)), add2(h, f));
}

// float64 as float pairs with the runs folded into a normalised float pair: no FP64 instruction
// until the sum is read (UP in pair form).  The low part is renormalised every two additions, not four (2% of
// the time of a wide product): mean errors of UP products stay 15-20% below the sweep's.
template <int NP> struct PackedF64SD {
    float2 hi[NP], lo[NP], thi[NP], tlo[NP];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int j = 0; j < NP; j++) hi[j] = lo[j] = thi[j] = tlo[j] = make_float2(0.0f, 0.0f);
    }
    __device__ __forceinline__ void add(const DF* v) {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            float2 s, e;
            two_sum2(hi[j], make_float2(v[2 * j].hi, v[2 * j + 1].hi), s, e);
            lo[j] = add2(lo[j], add2(e, make_float2(v[2 * j].lo, v[2 * j + 1].lo)));
            hi[j] = s;
        }
    }
    template <int N> __device__ __forceinline__ void add_block(const DF (*v)[2 * NP]) {
#pragma unroll
        for (int u = 0; u < N; u++) {
            add(v[u]);
            if (u & 1) settle();
        }
    }
    __device__ __forceinline__ void settle() {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            const float2 h = add2(hi[j], lo[j]);
            lo[j] = sub2(lo[j], sub2(h, hi[j]));
            hi[j] = h;
        }
    }
    __device__ __forceinline__ void flush() {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            df_add2(thi[j], tlo[j], hi[j], lo[j]);
            hi[j] = lo[j] = make_float2(0.0f, 0.0f);
        }
    }
    __device__ __forceinline__ void merge(const PackedF64SD& o) {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            df_add2(thi[j], tlo[j], o.thi[j], o.tlo[j]);
            df_add2(thi[j], tlo[j], o.hi[j], o.lo[j]);
        }
    }
    __device__ __forceinline__ PackedF64SD shfl_xor(int m) const {
        PackedF64SD r;
#pragma unroll
        for (int j = 0; j < NP; j++) {
            r.hi[j] = shfl_xor2(hi[j], m);
            r.lo[j] = shfl_xor2(lo[j], m);
            r.thi[j] = shfl_xor2(thi[j], m);
            r.tlo[j] = shfl_xor2(tlo[j], m);
        }
        return r;
    }
    // The sum as one float pair.
    __device__ __forceinline__ DF pair(int i) const {
        return df_add(DF{lane_of(thi[i >> 1], i), lane_of(tlo[i >> 1], i)}, DF{lane_of(hi[i >> 1], i), lane_of(lo[i >> 1], i)});
    }
    __device__ __forceinline__ F64Run get(int i) const {
        return {static_cast<double>(lane_of(thi[i >> 1], i)) + static_cast<double>(lane_of(tlo[i >> 1], i)),
                lane_of(hi[i >> 1], i), lane_of(lo[i >> 1], i)};
    }
};
template <> struct VecAcc<AddF64SD, 2> : PackedF64SD<1> {};
// One column: the pair form of the accumulator with an unused second half.
template <> struct VecAcc<AddF64SD, 1> : PackedF64SD<1> {
    using Base = PackedF64SD<1>;
    __device__ __forceinline__ VecAcc() = default;
    __device__ __forceinline__ VecAcc(const Base& b) : Base(b) {}
    template <int N> __device__ __forceinline__ void add_block(const DF (*v)[1]) {
        // two rows at a time, one in each half
#pragma unroll
        for (int u = 0; u < N; u += 2) {
            const DF w[2] = {v[u][0], v[u + 1][0]};
            Base::add(w);
            if ((u & 2) != 0) settle();
        }
    }
    __device__ __forceinline__ DF pair(int) const { return df_add(Base::pair(0), Base::pair(1)); }
    __device__ __forceinline__ F64Run get(int) const {
        const F64Run a = Base::get(0), b = Base::get(1);
        return {a.acc + b.acc + AddF64S::run_value(b), a.hi, a.lo};
    }
};

// Plain floats and doubles, grouped: the rows of a block as a tree, and (RUNS) blocks in runs, runs onto the sum.
// Error and time: pair_down_f32.cu.
template <class Op, int VW, bool RUNS> struct GroupedAcc {
    using S = typename Op::S;
    S run[VW], sum[RUNS ? VW : 1], held[RUNS ? VW : 1];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int i = 0; i < VW; i++) run[i] = S(0);
        if constexpr (RUNS) {
#pragma unroll
            for (int i = 0; i < VW; i++) sum[i] = S(0);
        }
    }
    template <int N> static __device__ __forceinline__ S tree(const S (*v)[VW], int i) {
        static_assert((N & (N - 1)) == 0, "a whole tree");
        S t[N];
#pragma unroll
        for (int u = 0; u < N; u++) t[u] = v[u][i];
#pragma unroll
        for (int n = N / 2; n > 0; n /= 2) {
#pragma unroll
            for (int u = 0; u < n; u++) t[u] = t[2 * u] + t[2 * u + 1];
        }
        return t[0];
    }
    template <int N> __device__ __forceinline__ void add_block(const S (*v)[VW]) {
#pragma unroll
        for (int i = 0; i < VW; i++) run[i] += tree<N>(v, i);
    }
    __device__ __forceinline__ void add_pairs(const S (*v)[VW]) { add_block<4>(v); }
    // Four rows whose sum waits for the next four's.
    __device__ __forceinline__ void hold_rows(const S (*v)[VW]) {
#pragma unroll
        for (int i = 0; i < VW; i++) held[i] = tree<4>(v, i);
    }
    __device__ __forceinline__ void add_rows(const S (*v)[VW]) {
#pragma unroll
        for (int i = 0; i < VW; i++) run[i] += held[i] + tree<4>(v, i);
    }
    __device__ __forceinline__ void add_held() {
#pragma unroll
        for (int i = 0; i < VW; i++) run[i] += held[i];
    }
    __device__ __forceinline__ void flush() {
        if constexpr (RUNS) {
#pragma unroll
            for (int i = 0; i < VW; i++) {
                sum[i] += run[i];
                run[i] = S(0);
            }
        }
    }
    // No more blocks: the sum is whole from here on.
    __device__ __forceinline__ void seal() {
        if constexpr (RUNS) {
#pragma unroll
            for (int i = 0; i < VW; i++) run[i] += sum[i];
        }
    }
    __device__ __forceinline__ void merge(const GroupedAcc& o) {
#pragma unroll
        for (int i = 0; i < VW; i++) run[i] += o.run[i];
    }
    __device__ __forceinline__ GroupedAcc shfl_xor(int m) const {
        GroupedAcc r;
#pragma unroll
        for (int i = 0; i < VW; i++) r.run[i] = Op::shfl_xor(run[i], m);
        return r;
    }
    __device__ __forceinline__ S get(int i) const { return run[i]; }
};
template <int VW> struct VecAcc<AddF32G, VW> : GroupedAcc<AddF32G, VW, true> {};
template <int VW> struct VecAcc<AddF64G, VW> : GroupedAcc<AddF64G, VW, true> {};
template <int VW> struct VecAcc<AddF64T, VW> : GroupedAcc<AddF64T, VW, false> {};

// float64 as float pairs in runs of four or eight rows, each run folded into a DFSum: a run's first row is its
// start, the pair is renormalised after four, and no FP64 instruction is needed at all (FP64 conversions and
// additions run at about two lanes per clock and SM).  A run's low parts are rounded relative to its sum,
// so the run's length sets the error: see pair_down_f64s.cu.
template <int NP> struct PackedF64ST {
    float2 hi[NP], lo[NP], t0[NP], t1[NP], t2[NP];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int j = 0; j < NP; j++) t0[j] = t1[j] = t2[j] = make_float2(0.0f, 0.0f);
    }
    __device__ __forceinline__ void start(const DF* v) {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            hi[j] = make_float2(v[2 * j].hi, v[2 * j + 1].hi);
            lo[j] = make_float2(v[2 * j].lo, v[2 * j + 1].lo);
        }
    }
    __device__ __forceinline__ void add(const DF* v) {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            float2 s, e;
            two_sum2(hi[j], make_float2(v[2 * j].hi, v[2 * j + 1].hi), s, e);
            lo[j] = add2(lo[j], add2(e, make_float2(v[2 * j].lo, v[2 * j + 1].lo)));
            hi[j] = s;
        }
    }
    __device__ __forceinline__ void settle() {
#pragma unroll
        for (int j = 0; j < NP; j++) {
            const float2 h = add2(hi[j], lo[j]);
            lo[j] = sub2(lo[j], sub2(h, hi[j]));
            hi[j] = h;
        }
    }
    __device__ __forceinline__ void fold() {  // (DFSum::fold)
#pragma unroll
        for (int j = 0; j < NP; j++) {
            float2 s, e, f, g;
            two_sum2(t0[j], hi[j], s, e);
            t0[j] = s;
            two_sum2(t1[j], lo[j], s, f);
            two_sum2(s, e, t1[j], g);
            t2[j] = add2(t2[j], add2(f, g));
        }
    }
    // Four rows that start a run, and four more.
    __device__ __forceinline__ void start_rows(const DF (*v)[2 * NP]) {
        start(v[0]);
#pragma unroll
        for (int u = 1; u < 4; u++) add(v[u]);
        settle();
    }
    __device__ __forceinline__ void add_rows(const DF (*v)[2 * NP]) {
#pragma unroll
        for (int u = 0; u < 4; u++) add(v[u]);
    }
    __device__ __forceinline__ DFSum get(int i) const {
        return {lane_of(t0[i >> 1], i), lane_of(t1[i >> 1], i), lane_of(t2[i >> 1], i)};
    }
};
template <> struct VecAcc<AddF64ST, 2> : PackedF64ST<1> {};
// One column: two rows at a time, one in each half.
template <> struct VecAcc<AddF64ST, 1> : PackedF64ST<1> {
    using Base = PackedF64ST<1>;
    __device__ __forceinline__ void start_rows(const DF (*v)[1]) {
        const DF a[2] = {v[0][0], v[1][0]}, b[2] = {v[2][0], v[3][0]};
        start(a);
        add(b);
    }
    __device__ __forceinline__ void add_rows(const DF (*v)[1]) {
        const DF a[2] = {v[0][0], v[1][0]}, b[2] = {v[2][0], v[3][0]};
        add(a);
        add(b);
    }
    __device__ __forceinline__ DFSum get(int) const {
        DFSum a = Base::get(0);
        const DFSum b = Base::get(1);
        a.fold(DF{b.t0, b.t1});
        a.t2 = __fadd_rn(a.t2, b.t2);
        return a;
    }
};

// Every addition normalised: four rows as a two-level tree, then onto the sum.
template <int NP> struct PackedF64SN {
    float2 hi[NP], lo[NP];
    __device__ __forceinline__ void zero() {
#pragma unroll
        for (int j = 0; j < NP; j++) hi[j] = lo[j] = make_float2(0.0f, 0.0f);
    }
    template <int N> __device__ __forceinline__ void add_block(const DF (*v)[2 * NP]) {
        static_assert(N % 4 == 0, "block of whole trees");
#pragma unroll
        for (int u = 0; u < N; u += 4) {
#pragma unroll
            for (int j = 0; j < NP; j++) {
                float2 h[4], l[4];
#pragma unroll
                for (int t = 0; t < 4; t++) {
                    h[t] = make_float2(v[u + t][2 * j].hi, v[u + t][2 * j + 1].hi);
                    l[t] = make_float2(v[u + t][2 * j].lo, v[u + t][2 * j + 1].lo);
                }
                df_add2(h[0], l[0], h[1], l[1]);
                df_add2(h[2], l[2], h[3], l[3]);
                df_add2(h[0], l[0], h[2], l[2]);
                df_add2(hi[j], lo[j], h[0], l[0]);
            }
        }
    }
    __device__ __forceinline__ void flush() {}
    __device__ __forceinline__ void merge(const PackedF64SN& o) {
#pragma unroll
        for (int j = 0; j < NP; j++) df_add2(hi[j], lo[j], o.hi[j], o.lo[j]);
    }
    __device__ __forceinline__ PackedF64SN shfl_xor(int m) const {
        PackedF64SN r;
#pragma unroll
        for (int j = 0; j < NP; j++) {
            r.hi[j] = shfl_xor2(hi[j], m);
            r.lo[j] = shfl_xor2(lo[j], m);
        }
        return r;
    }
    __device__ __forceinline__ DF pair(int i) const { return {lane_of(hi[i >> 1], i), lane_of(lo[i >> 1], i)}; }
    __device__ __forceinline__ F64Run get(int i) const { return {0.0, lane_of(hi[i >> 1], i), lane_of(lo[i >> 1], i)}; }
};
template <> struct VecAcc<AddF64SN, 2> : PackedF64SN<1> {};
template <> struct VecAcc<AddF64SN, 1> : PackedF64SN<1> {
    __device__ __forceinline__ VecAcc() = default;
    template <int N> __device__ __forceinline__ void add_block(const DF (*v)[1]) {
        DF w[N / 2][2];
#pragma unroll
        for (int u = 0; u < N / 2; u++) {
            w[u][0] = v[2 * u][0];
            w[u][1] = v[2 * u + 1][0];
        }
        PackedF64SN<1>::template add_block<N / 2>(w);
    }
    __device__ __forceinline__ DF pair(int) const { return df_add(PackedF64SN<1>::pair(0), PackedF64SN<1>::pair(1)); }
    __device__ __forceinline__ F64Run get(int) const {
        const DF r = pair(0);
        return {0.0, r.hi, r.lo};
    }
};

}  // namespace grgx
