// tracer_cell.cuh - the tracer update of one cell (moist.jl:1479-1515) on two lanes of a warp.
//
// The update is adv_x + adv_z and diff_x + diff_z, two halves of the same shape: two limited face
// fluxes (moist.jl:850-945), their difference over a length, and two face gradients. A warp
// holds WROWS = 16 rows of the sweep: lane r evaluates the x half of row r, lane r + 16 its z half, in
// one instruction stream, and the halves meet by two shuffles, after which both lanes hold the
// new value. What bounds the sweeps is the latency of this function along the Gauss-Seidel chain
// (a warp alone on its scheduler) and its instruction count (several warps): per row of 16 cells
// and step this is about half the instructions and half the dependent length of one lane doing a
// whole cell.
//
// Every expression keeps the reference's operation order. Differences between the halves become
// lane constants that leave each half's value bit for bit: the x half's centred face value
// 0.5 (a + b) is (a 1 + b 1) / 2, its limited value s_p1 + half against the z half's s_p1 - half is a
// flipped sign bit, its faces never clamp and never vanish.
#pragma once

#include "fastdiv.cuh"
#include "kernels.cuh"

namespace moist {

constexpr int WROWS = 16;  // rows of a warp

// lane constants: the p face is i+1/2 (x half) or k+1/2 (z half), the m face i-1/2 or k-1/2
template <class T>
struct HalfRow {
    T h;                             // dx or dz[k]
    T wa_p, wb_p, sum_p;             // centred value of the p face: (s_0 wb + s_p1 wa) / sum
    T wa_m, wb_m, sum_m;
    T den_p, den_m;                  // distance of the cell centres around the face
    Rcp<T> rh, rsum_p, rsum_m, rden_p, rden_m;
    T kappa, EPS, dt;
    unsigned neg_sign;               // the sign bit of the limiter's half step for a negative velocity
    unsigned zero_p, zero_m;         // faces without flux (k = ke, k = 0)
    unsigned p_at0, p_atn, m_at0, m_atn;  // z faces that clamp: lower cell 0 (upward flow), nz-2 (downward)
};

// constants of row k for the half `z`; rows outside the domain get harmless ones
template <class T>
__device__ __forceinline__ HalfRow<T> half_row(const DevParams<T>& p, int k, bool z, T dt_stage) {
    const int nz = p.nz, ke = nz - 1;
    const bool in = k < nz;
    HalfRow<T> w;
    w.kappa = p.kappa;
    w.EPS = p.EPS;
    w.dt = dt_stage;
    w.neg_sign = z ? 0x80000000u : 0u;
    if (z) {
        const T dz_k = in ? p.dz[k] : T(1), dz_kp1 = k < ke ? p.dz[k + 1] : T(1),
                dz_km1 = (in && k > 0) ? p.dz[k - 1] : T(1);
        const T z_k = in ? p.z[k] : T(0), z_kp1 = k < ke ? p.z[k + 1] : T(1), z_km1 = (in && k > 0) ? p.z[k - 1] : T(-1);
        w.h = dz_k;
        w.wa_p = dz_k;
        w.wb_p = dz_kp1;
        w.sum_p = dz_k + dz_kp1;
        w.wa_m = dz_km1;
        w.wb_m = dz_k;
        w.sum_m = dz_km1 + dz_k;
        w.den_p = z_kp1 - z_k;
        w.den_m = z_k - z_km1;
    } else {
        w.h = w.den_p = w.den_m = p.dx;
        w.wa_p = w.wb_p = w.wa_m = w.wb_m = T(1);
        w.sum_p = w.sum_m = T(2);
    }
    w.rh = FastDiv<T>::prep(w.h);
    w.rsum_p = FastDiv<T>::prep(w.sum_p);
    w.rsum_m = FastDiv<T>::prep(w.sum_m);
    w.rden_p = FastDiv<T>::prep(w.den_p);
    w.rden_m = FastDiv<T>::prep(w.den_m);
    w.zero_p = z && k == ke;
    w.zero_m = z && k == 0;
    w.p_at0 = z && k == 0;
    w.p_atn = z && k == nz - 2;
    w.m_at0 = z && k == 1;
    w.m_atn = z && k == nz - 1;
    return w;
}

// 0.5 koren(r_num / r_den), with r = 1 where |r_den| < EPS (moist.jl:846): half of
// max(0, min(2 r, min((1 + 2 r) / 3, 2))) is max(0, min(r, min((1 + 2 r) / 6, 1))), exactly (half a
// quotient by 3 is the quotient by 6, 2 r is exact). Float has the minima as single instructions. In
// double each is several, on the chain: there the interval of r is read from its bits while the
// division is under way, and one selection follows: 0 for r <= 0, r up to 1/4, 1 from 5/2 on and
// (1 + 2 r) / 6 between them, of the rounded values too (rounding is monotone, and the two sides meet
// exactly at 1/4 and 5/2); NaN takes the division's branch. The walk of a Float64 tile (200 x 100):
// 41.8 -> 31.0 us with this, the scaled denominators and the shorter reciprocal. The same in Float32
// made the sweeps 1 to 4 % slower.
template <class D, class T>
__device__ __forceinline__ T half_koren(T r_num, T r_den, T EPS, bool& bad) {
    const bool one = fabs(r_den) < EPS;
    const T ratio = D::ratio(r_num, r_den, one, bad);
    if constexpr (sizeof(T) == 4) {
        const T r = one ? T(1) : ratio;
        return jmax_f(T(0), jmin_f(r, jmin_f(D::div6(fma_t(T(2), r, T(1))), T(1))));
    } else {
        constexpr unsigned SIGN = 0x80000000u, INF = 0x7ff00000u, QUARTER = 0x3fd00000u, B25 = 0x40040000u;
        const unsigned x = (unsigned)__double2hiint(ratio);
        const bool low = x - SIGN <= INF, small = x < QUARTER, big = x - B25 <= INF - B25;  // -0 and -inf are low
        const T e = one ? T(0.5) : (low ? T(0) : (small ? ratio : T(1)));
        const T d = D::div6(fma_t(T(2), ratio, T(1)));
        return (one | low | small | big) ? e : d;
    }
}

// the limited flux through one face (moist.jl:850-945). CEN: cen and clamp are formed and a face may
// select them; elsewhere every face has |vel| > EPS and none clamps.
template <class D, bool CEN, class T>
__device__ __forceinline__ T half_flux(const HalfRow<T>& w, T vel, T s_m1, T s_0, T s_p1, T s_p2, T cen, T clamp,
                                       unsigned at0, unsigned atn, bool& bad) {
    const bool pos = vel > w.EPS;
    const unsigned m = pos ? 0u : 0x80000000u;
    const T up = pos ? s_0 : s_p1;
    const T r_num = flip(s_p1 - s_0, m);  // the sign of a zero does not matter to the limiter
    const T r_den = up - (pos ? s_m1 : s_p2);
    const T half = half_koren<D>(r_num, r_den, w.EPS, bad) * r_den;
    T face = up + flip(half, m & w.neg_sign);
    if constexpr (CEN) {
        const bool neg = vel < -w.EPS, cl = (pos & (at0 != 0u)) | (neg & (atn != 0u));
        const T other = cl ? clamp : cen;
        face = ((pos | neg) & !cl) ? face : other;
    }
    return face * vel;
}

// this lane's half: advection and diffusion terms. CEN: form the centred face values, which only
// faces with |vel| <= EPS and clamping faces select, and set the faces without flux to zero (the
// sweeps know where there are none of these). (m2, m1, c, p1, p2) are the five values along
// the half's direction, m2 and m1 updated; cl_p / cl_m the clamp quotients lin / (+-vel dt).
template <class D, bool CEN, class T>
__device__ __forceinline__ void half_cell(const HalfRow<T>& w, T m2, T m1, T c, T p1, T p2, T vel_p,
                                          T vel_m, T rf_p, T rf_m, T cl_p, T cl_m, T& adv, T& diff, bool& bad) {
    T cen_p = T(0), cen_m = T(0), clamp_p = T(0), clamp_m = T(0);
    if constexpr (CEN) {
        cen_p = D::cdiv(c * w.wb_p + p1 * w.wa_p, w.sum_p, w.rsum_p);
        cen_m = D::cdiv(m1 * w.wb_m + c * w.wa_m, w.sum_m, w.rsum_m);
        clamp_p = jmin_f(cen_p, cl_p);
        clamp_m = jmin_f(cen_m, cl_m);
        bad |= !(fabs(cen_p) <= DivRange<T>::MAX) || !(fabs(cen_m) <= DivRange<T>::MAX);  // a minimum could hide it
    }
    T f_p = half_flux<D, CEN>(w, vel_p, m1, c, p1, p2, cen_p, clamp_p, w.p_at0, w.p_atn, bad);
    T f_m = half_flux<D, CEN>(w, vel_m, m2, m1, c, p1, cen_m, clamp_m, w.m_at0, w.m_atn, bad);
    T d_p = D::cdiv(rf_p * (p1 - c), w.den_p, w.rden_p);
    T d_m = D::cdiv(rf_m * (c - m1), w.den_m, w.rden_m);
    if constexpr (CEN) {  // the lowest and highest rows clamp as well
        f_p = sel_u(w.zero_p, T(0), f_p);
        f_m = sel_u(w.zero_m, T(0), f_m);
        d_p = sel_u(w.zero_p, T(0), d_p);
        d_m = sel_u(w.zero_m, T(0), d_m);
    }
    adv = D::cdiv(f_p - f_m, w.h, w.rh);
    diff = D::cdiv(w.kappa * (d_p - d_m), w.h, w.rh);
}

// the whole cell of both lanes' row: new rho_q and s = rho_q / rho. Every lane of the warp calls it.
template <class D, bool CEN, class T>
__device__ __forceinline__ void two_lane_cell(const HalfRow<T>& w, T m2, T m1, T c, T p1, T p2, T vel_p, T vel_m, T rf_p,
                                              T rf_m, T cl_p, T cl_m, T q0, T dph, T rho, T rrho, T& q, T& s,
                                              bool& bad) {
    T adv, diff;
    half_cell<D, CEN>(w, m2, m1, c, p1, p2, vel_p, vel_m, rf_p, rf_m, cl_p, cl_m, adv, diff, bad);
    const T adv_o = __shfl_xor_sync(0xffffffffu, adv, WROWS), diff_o = __shfl_xor_sync(0xffffffffu, diff, WROWS);
    const T advection = -(adv + adv_o);
    const T diffusion = diff + diff_o;
    q = q0 + w.dt * (advection + diffusion + dph);
    s = D::quot(q, rho, rrho, bad);
    bad |= !(fabs(s) <= DivRange<T>::MAX);
}

}  // namespace moist
