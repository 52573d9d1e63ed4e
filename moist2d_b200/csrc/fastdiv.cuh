// fastdiv.cuh - branch-free, correctly rounded division for the hot loops.
//
// CUDA's IEEE division ends every quotient with a range check and a branch to a slow path (very
// slow for subnormal results), so consecutive divisions cannot overlap and the code between them
// cannot be scheduled together: a tracer cell of ~25 such divisions is ~1800 cycles of dependent
// latency, and the Gauss-Seidel tracer sweep walks long chains of cells. In its place:
//   FastDiv<T> (tracer cell, column solve): remainder corrections in the type's own precision; what
//       it cannot round exactly is reported and the caller repeats with IeeeDiv<T>;
//   div64 (slow tendencies): RN32(RN64(a y)) with a tabulated y = 1/b in double precision, the IEEE
//       quotient of floats but for ties in the subnormal range, which a guard word reports;
//   quotient_proven (acoustic substep): an exact test of a corrected double quotient, beside the
//       recurrence.
// tests/fastdiv_check.cu, tests/celldiv_check.cu and tests/quotient_check.cu compare them with IEEE division on
// the GPU, over all numerators for the model's denominators and on random bit patterns of every class.
#pragma once

#include <cuda_runtime.h>

#include "moist_math.h"

namespace moist {

// The sign of a zero result: for a nonzero quotient q and q0 (two roundings of the same value)
// share their sign, so OR-ing the sign bit of q0 into q only changes a zero.
__device__ __forceinline__ float with_sign_of(float q, float q0) {
    return __int_as_float(__float_as_int(q) | (__float_as_int(q0) & (int)0x80000000));
}

// A select the compiler cannot turn into a branch: both operands are always computed, so the
// independent parts of a cell update stay in one basic block and overlap.
__device__ __forceinline__ double sel_u(unsigned c, double x, double y) { return c != 0 ? x : y; }
__device__ __forceinline__ float sel_u(unsigned c, float x, float y) {  // c != 0 ? x : y
    float r;
    asm("{\n\t.reg .pred p;\n\tsetp.ne.u32 p, %1, 0;\n\tselp.f32 %0, %2, %3, p;\n\t}"
        : "=f"(r) : "r"(c), "f"(x), "f"(y));
    return r;
}

__device__ __forceinline__ bool same_bits(float x, float y) { return __float_as_uint(x) == __float_as_uint(y); }
__device__ __forceinline__ bool same_bits(double x, double y) { return __double_as_longlong(x) == __double_as_longlong(y); }

// the sign of x flipped where the bit `m` (0 or 0x80000000) is set
__device__ __forceinline__ float flip(float x, unsigned m) { return __uint_as_float(__float_as_uint(x) ^ m); }
__device__ __forceinline__ double flip(double x, unsigned m) {
    return __hiloint2double(__double2hiint(x) ^ (int)m, __double2loint(x));
}

// Julia's min / max (NaN-propagating, -0 < +0) as single PTX instructions
__device__ __forceinline__ float jmin_f(float a, float b) {
    float r;
    asm("min.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ float jmax_f(float a, float b) {
    float r;
    asm("max.NaN.f32 %0, %1, %2;" : "=f"(r) : "f"(a), "f"(b));
    return r;
}
__device__ __forceinline__ double jmin_f(double a, double b) { return mm::jmin(a, b); }
__device__ __forceinline__ double jmax_f(double a, double b) { return mm::jmax(a, b); }

// ---- FP64-reciprocal division: RN32(a/b) = RN32(RN64(a * y)) for y = 1/b to within 2^-51
//
// For floats a, b whose quotient is not a float itself, a/b lies at a relative distance of at
// least 2^-48 from every float rounding boundary (a midpoint between neighbouring floats, or
// the overflow threshold): with A, B the integer significands, a boundary M near A/B gives
// |A/B - M| >= 1/(B 2^25), and in the subnormal range the distance is larger still. A normal
// quotient is never exactly a boundary (that needs 25 significant bits from a product of
// B <= 24 bits and A); a subnormal one can be, e.g. (3 * 2^-149) / 6 = 2^-150. The product a*y
// rounded to double is within 2^-52 + 2^-51 of a/b (the double product neither underflows nor
// overflows), so it lies on the same side of every boundary and rounding it to float gives the
// IEEE quotient, except for those exact subnormal ties. Every quotient q in 0 < |q| <= 2^-126
// is therefore reported through a guard word (subnormal_guard), and the caller recomputes such
// a cell with IEEE division; zeros, infinities and NaN come out as IEEE division gives them.
__device__ __forceinline__ float div64(float a, double y) { return __double2float_rn((double)a * y); }

// div64 exact for every input: a quotient below 2^-125 in magnitude (float spacing 2^-149) is
// rounded explicitly on that grid. w = p 2^149 is the quotient in grid units, within 2^-28 of
// the exact value; an exact quotient that is not a tie lies at least 2^-25 from every
// half-integer (the nonzero integer |A 2^e - B (2k+1)| over 2B, with B >= 2^23 since b is
// normal whenever a/b < 2^-125), so |w - fl - 1/2| < 2^-26 detects the ties, which go to the
// even neighbour; every other w rounds to its nearest integer. The sign of a zero is p's.
__device__ __forceinline__ float div64x(float a, double y) {
    const double p = (double)a * y;
    const float qn = __double2float_rn(p);
    const double w = p * 0x1p149;
    const double fl = floor(w);
    const bool tie = fabs((w - fl) - 0.5) < 0x1p-26;
    const double even = (fl - 2.0 * floor(fl * 0.5)) == 0.0 ? fl : fl + 1.0;
    const float qs = with_sign_of((float)((tie ? even : rint(w)) * 0x1p-149), qn);
    return fabs(p) < 0x1p-125 ? qs : qn;
}

// fold q into the guard word g (start from ~0u): afterwards g < 2^24 iff some q had
// 0 < |q| <= 2^-126 (the doubled bit pattern of 2^-126 is 2^24; zero maps to ~0u)
__device__ __forceinline__ void subnormal_guard(unsigned& g, float q) { g = min(g, (__float_as_uint(q) << 1) - 1u); }
__device__ __forceinline__ bool guard_hit(unsigned g) { return g < (1u << 24); }

// 1/b to within 2^-51 relative (b finite and nonzero): the hardware approximation and two
// Newton steps e = 1 - b y, y += y e in double precision
__device__ __forceinline__ double rcp64(float b) {
    const double bd = (double)b;
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(bd));
    double e = __fma_rn(-bd, y, 1.0);
    y = __fma_rn(y, e, y);
    e = __fma_rn(-bd, y, 1.0);
    return __fma_rn(y, e, y);
}

// Division by the double reciprocal: cdiv(a, b, y, g) with y = 1/b prepared once is what the slow
// tendencies do (div64 and the guard); the variable denominator (vdiv, rcp64) and the explicit rounding
// (Div64X, div64x) are compared with IEEE division by tests/fastdiv_check.cu and not used by any
// kernel. g is the subnormal guard word.
struct Div64 {  // FP64 reciprocal: exact for every input but subnormal ties, which g reports
    using R = double;
    __device__ __forceinline__ static R rcp(float b) { return 1.0 / (double)b; }
    __device__ __forceinline__ static float cdiv(float a, float, R y, unsigned& g) {
        const float q = div64(a, y);
        subnormal_guard(g, q);
        return q;
    }
    __device__ __forceinline__ static float vdiv(float a, float b, unsigned& g) {
        const float q = div64(a, rcp64(b));
        subnormal_guard(g, q);
        return q;
    }
};
struct Div64X {  // FP64 reciprocal with explicit rounding of subnormal quotients: exact for every input
    using R = double;
    __device__ __forceinline__ static R rcp(float b) { return 1.0 / (double)b; }
    __device__ __forceinline__ static float cdiv(float a, float, R y, unsigned&) { return div64x(a, y); }
    __device__ __forceinline__ static float vdiv(float a, float b, unsigned&) { return div64x(a, rcp64(b)); }
};

// ---- division in the type's own arithmetic: remainder corrections on a reciprocal
//
// Let q0 be within one ulp of a/b. Its remainder a - b q0 is then a float (the FMA forms it
// exactly), and RN(q0 + (a - b q0) RN(1/b)) = RN(a/b) (P. Markstein, IBM J. Res. Dev. 34, 1990;
// the quotient theorem of Muller et al., Handbook of Floating-Point Arithmetic). The remainder
// must not underflow: it is formed from the numerator and the denominator scaled by UP (both exact,
// and off the dependent path), and the last FMA takes it back with RN(1/b) / UP onto the unscaled
// q0, so a subnormal quotient too is rounded once, onto its own grid. There the argument holds but for exact ties (the rounding
// error of 1/b decides them): a tie is |remainder| = b times half a grid unit. cdiv sends it to the
// even neighbour (the tails at the edges of clouds fall through the subnormal range within a few
// cells, where every hundredth or so quotient by 100 or 250 is one); in quot and ratio, whose
// denominators have long significands, it sets `bad`.
//   prepared b (cdiv): q0 = RN(a d + RN(a l)) with d + l = 1/b to 2^-40, and one correction;
//   variable b: with y0 = 1/b to about one ulp, q0 = RN(a y0) is within a few ulps, one correction
//   with y0 makes it one of the two values around a/b, a second one, with RN(1/b) formed
//   meanwhile, RN(a/b).
// d is 1/b rounded down, so that both terms of q0 and the correction of a zero keep the sign of a
// zero numerator (b > 0). What leaves the admitted ranges ends as a non-finite result or sets
// `bad`, never as a wrong finite one: a prepared denominator outside [LO, HI] has NaN
// reciprocals, |a| UP overflows to an infinity that the correction turns into an infinity or NaN, a variable denominator above BIG sets `bad`. The sweeps check `bad` and the
// finiteness of their results once per tile or sweep and repeat it with IeeeDiv.
// tests/celldiv_check.cu compares every primitive with IEEE division on the GPU: all 2^32 numerators for
// the model's denominators, all 2^32 denominators for the reciprocal, and random bit patterns.
//
// Against a multiplication by the reciprocal in double precision (Div64) this leaves out the two
// conversions of every quotient, which an SM issues at 16 lanes a cycle (a quarter of a warp's
// FMA rate per scheduler); against CUDA's division it has no branch.
template <class T>
struct Rcp {        // reciprocal of a prepared denominator b
    T d, l, n;      // 1/b rounded down, the rest 1/b - d, and RN(1/b) / UP
    T tie;          // the remainder of an exact subnormal tie (-1 for a power of two)
};

template <class T>
struct DivRange;
template <>
struct DivRange<float> {
    static constexpr float UP = 0x1p64f, DOWN = 0x1p-64f, TIE = 0x1p-86f;  // TIE = 2^-150 UP
    static constexpr float LO = 0x1p-40f, HI = 0x1p40f, BIG = 0x1p60f, MAX = 0x1.fffffep127f;
};
template <>
struct DivRange<double> {
    static constexpr double UP = 0x1p200, DOWN = 0x1p-200, TIE = 0x1p-875;  // TIE = 2^-1075 UP
    static constexpr double LO = 0x1p-100, HI = 0x1p100, BIG = 0x1p800, MAX = 0x1.fffffffffffffp1023;
};

__device__ __forceinline__ float fma_t(float a, float b, float c) { return __fmaf_rn(a, b, c); }
__device__ __forceinline__ bool odd(float x) { return (__float_as_uint(x) & 1u) != 0u; }
__device__ __forceinline__ bool odd(double x) { return (__double_as_longlong(x) & 1ll) != 0; }
__device__ __forceinline__ double fma_t(double a, double b, double c) { return __fma_rn(a, b, c); }

__device__ __forceinline__ float rcp_rd(float b) { return __frcp_rd(b); }
__device__ __forceinline__ double rcp_rd(double b) { return __drcp_rd(b); }

// 1/b of a variable denominator: y0 to about one ulp and RN(1/b). Float: y0 is the hardware
// approximation and one Newton step gives RN(1/b), checked against IEEE division for every |b| in
// [2^-125, 2^125]. Double: the cubic step y (1 + e + e e) on the approximation's 20 bits or more
// reaches one ulp, and a Newton step on it gives RN(1/b) unless b's significand is all ones
// (Markstein), which sets bad.
__device__ __forceinline__ float rcp_rn(float b, float& y0, bool&) {
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y0) : "f"(b));
    return __fmaf_rn(y0, __fmaf_rn(-b, y0, 1.0f), y0);
}
__device__ __forceinline__ double rcp_rn(double b, double& y0, bool& bad) {
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));
    const double e = __fma_rn(-b, y, 1.0);
    y0 = __fma_rn(y, __fma_rn(e, e, e), y);
    bad |= ((unsigned long long)__double_as_longlong(b) << 12) == 0xfffffffffffff000ull;
    return __fma_rn(y0, __fma_rn(-b, y0, 1.0), y0);
}

template <class T>
struct FastDiv : DivRange<T> {
    using DR = DivRange<T>;
    __device__ __forceinline__ static Rcp<T> prep(T b) {
        if (!(b >= DR::LO && b <= DR::HI)) {
            const T nan = T(0) / T(0);
            return {nan, nan, nan, nan};
        }
        const T y = T(1) / b, d = rcp_rd(b), e = fma_t(-b, d, T(1));  // 1 - b d is exact
        return {d, e * y, y * DR::DOWN, e == T(0) ? T(-1) : b * DR::TIE};
    }
    // RN(1/b) of a prepared denominator for quot()
    __device__ __forceinline__ static T prep1(T b) { return b >= DR::LO && b <= DR::HI ? T(1) / b : T(0) / T(0); }
    __device__ __forceinline__ static T cdiv(T a, T b, const Rcp<T>& y) {
        const T q0 = fma_t(a, y.d, a * y.l);
        const T rn = fma_t(b * DR::UP, q0, -(a * DR::UP));  // negated: +0 for a zero of either sign
        // on a tie the correction with a slightly larger reciprocal reaches the other neighbour
        const T other = fma_t(-rn, y.n * T(1.0000305), q0);
        return fabs(rn) == y.tie ? (odd(q0) ? other : q0) : fma_t(-rn, y.n, q0);
    }
    // a / b with y = RN(1/b) and y0 near it
    __device__ __forceinline__ static T twice(T a, T b, T y0, T y, T tie, bool& bad) {
        const T as = -(a * DR::UP), bs = b * DR::UP;
        T q = a * y0;
        q = fma_t(-fma_t(bs, q, as), y0 * DR::DOWN, q);
        const T rn = fma_t(bs, q, as);
        bad |= fabs(rn) == tie;
        return fma_t(-rn, y * DR::DOWN, q);
    }
    // a / b with y = prep1(b)
    __device__ __forceinline__ static T quot(T a, T b, T y, bool& bad) { return twice(a, b, y, y, b * DR::TIE, bad); }
    // a / b for a variable b > 0; a result that is not finite sets bad
    __device__ __forceinline__ static T quot_var(T a, T b, bool& bad) {
        T y0;
        const T y = rcp_rn(b, y0, bad);
        const T q = twice(a, b, y0, y, b * DR::TIE, bad);
        bad |= b > DR::BIG || !(fabs(q) <= DR::MAX);
        return q;
    }
    // the limiter ratio a / b, not used where `one` (the sign of a zero is not kept for b < 0: the
    // limiter takes both zeros to +0)
    __device__ __forceinline__ static T ratio(T a, T b, bool one, bool& bad) {
        const T ab = fabs(b);
        bool refuse = ab > DR::BIG;
        T y0;
        const T y = rcp_rn(b, y0, refuse);
        const T q = twice(a, b, y0, y, ab * DR::TIE, refuse);
        bad |= !one && refuse;
        return q;
    }
    // (1 + 2 r) / 6: the numerator is 0 or at least 2^-24 (2^-53) in magnitude. 1/6 as the sum of two
    // values of the type, good to twice its precision: a quotient by 6 that is no tie lies a twelfth
    // of an ulp or more from every rounding boundary, and there are no ties but subnormal ones.
    __device__ __forceinline__ static T div6(T a) {
        constexpr T yh = T(1) / T(6);  // RN(1/6), and the rest exactly (1 - 6 yh) / 6
        constexpr T yl = sizeof(T) == 4 ? T(1.0 / 6.0 - (double)yh) : yh * T(0x1p-54);
        return fma_t(a, yh, a * yl);
    }
};

// the same interface with IEEE division
template <class T>
struct IeeeDiv {
    __device__ __forceinline__ static T cdiv(T a, T b, const Rcp<T>&) { return a / b; }
    __device__ __forceinline__ static T quot(T a, T b, T, bool&) { return a / b; }
    __device__ __forceinline__ static T quot_var(T a, T b, bool&) { return a / b; }
    __device__ __forceinline__ static T ratio(T a, T b, bool, bool&) { return a / b; }
    __device__ __forceinline__ static T div6(T a) { return a / T(6); }
};

// ---- exact test of a double quotient
//
// Let q1 be near a/b: the acoustic substep forms it from y = RN(1/b) with one correction by the
// remainder, q1 = RN(q0 + (a - b q0) y), which is the correctly rounded quotient in all but rare cases
// (Markstein, IBM J. Res. Dev. 34, 1990). When q1 lies within one ulp of a/b, the remainder
// r1 = a - b q1 is a double and the FMA forms it exactly (no underflow for the operand ranges admitted
// below), and |r1| < |b| u/2, with u the smaller of the two ulps around q1 (the ulp below a power of
// two is half the one above), says that a/b is nearer to q1 than to the midpoint towards either
// neighbour, i.e. q1 = RN(a/b). |b| u/2 is a power-of-two multiple of b, hence exact. When q1 is farther
// than one ulp the computed |r1| is at least RN(|b| u) = 2 (|b| u/2), so the test fails. It also fails
// where the operands leave 2^-960 <= |a| <= 2^1000, 2^-1000 <= |b| <= 2^1000 (non-finite values
// included): the caller then divides again with IEEE division.
__device__ __forceinline__ bool quotient_proven(double a, double b, double q1) {
    const double r1 = fma(-b, q1, a);
    const unsigned long long bits = (unsigned long long)__double_as_longlong(q1) & 0x7fffffffffffffffULL;
    const long long e = (long long)(bits >> 52);                                   // biased exponent of q1
    const long long he = e - 53 - ((bits & 0xfffffffffffffULL) == 0 ? 1 : 0);  // half of the smaller ulp
    const double half_u = __longlong_as_double((he < 1 ? 1LL : he) << 52);
    const double aa = fabs(a), ab = fabs(b);
    const bool in_range = aa >= 0x1p-960 && aa <= 0x1p1000 && ab >= 0x1p-1000 && ab <= 0x1p1000 && he >= 1;
    return in_range && fabs(r1) < ab * half_u;
}

}  // namespace moist
