// Model C device arithmetic shared by the step kernels, written in the
// reference's operand order.  Include only from translation units compiled
// with -fmad=false (see lg_kernels.cu).
#pragma once

#include <algorithm>
#include <cmath>
#include <cstring>
#include <limits>

#include "lg_common.cuh"
#include "lg_kernels.h"
#include "lg_quotient.cuh"

namespace lg {

template <class T>
struct MC {
    T lambda, d_thermal, a_bar, eps_prime, tol, f_a_bar, f_eps_prime, f_a12, f_tol, inv_h2_flux, ih0, ih1;
    T c_far, inv_c_far;  // a_bar * a_bar, the far-field mobility divisor, and RN(1 / c_far)
    unsigned far_face;    // face and centre keys below these are flat for certain (far_below)
    unsigned far_center;
    unsigned quotient_span;  // of the divisors that the faces' quotients take (quotient_span_of)
    unsigned safe_below;     // gradient keys below it are in that range (safe_below_of)
};

// The high half of a non-negative double, or the bits of a non-negative
// float: an unsigned number ordered as the values are, with every NaN above
// them all (one whose sign bit is set, as an invalid operation leaves it in a
// double, too).
__host__ __device__ __forceinline__ unsigned order_key(double s) { return high_word(s); }
__host__ __device__ __forceinline__ unsigned order_key(float s) {
#ifdef __CUDA_ARCH__
    return __float_as_uint(s);
#else
    unsigned b;
    memcpy(&b, &s, sizeof b);
    return b;
#endif
}

// The far field (|grad|^4 <= tol, in the reference's rounding) decided
// without its rounding: every |grad|^2 whose key is below the limit is below
// sqrt(tol) by more than any rounding of the sum and its square.  A limit of
// zero: none.  far_center is the limit for 4 |grad|^2, the sum of the whole
// differences' squares; no limit reaches the keys of infinity and NaN.
template <class T>
inline unsigned far_below(T tol, bool center) {
    if (!(tol > T(0))) return 0;
    const T s = std::sqrt(tol) * (T(1) - (sizeof(T) == 8 ? T(0x1p-40) : T(0x1p-20)));
    const unsigned two = 2u << (sizeof(T) == 8 ? 20 : 23);  // two binades
    return std::min(order_key(s) + (center ? two : 0u), order_key(std::numeric_limits<T>::infinity()));
}

// The quotients take the shared reciprocal for parameters as ordinary as
// these: a face's divisor |grad|^4 in [2^-900, 2^60) then keeps its first
// numerator e' (dx^4 + dy^4), at least half e' |grad|^4, and both quotients in
// quotient_rn's range, so that only a tiny second numerator is left to test,
// and the mobility's divisor a^2 stays below 2^60.  Others divide.
template <class T>
inline unsigned quotient_span_of(const MC<T>& m) {
    auto within = [](T e, T most) { return std::fabs(e) >= T(0x1p-50) && std::fabs(e) <= most; };
    auto none_or = [&](T e, T most) { return e == T(0) || within(e, most); };
    return none_or(m.eps_prime, T(0x1p10)) && none_or(m.f_eps_prime, T(0x1p10)) && none_or(m.f_a12, T(0x1p40)) &&
                   within(m.a_bar, T(0x1p18)) && within(m.f_a_bar, T(0x1p18))
               ? kQuotientSpan
               : 0;
}

// Passes whose gradients' keys are all below safe_below have every divisor in
// that range: |grad|^2 < 2^29, and a non-flat |grad|^4 is above the
// tolerances, which must not be tiny themselves (else no pass is safe).
template <class T>
inline unsigned safe_below_of(const MC<T>& m) {
    const bool tiny = !(m.f_tol >= T(0x1p-100) && m.tol >= T(0x1p-100));
    return tiny || m.quotient_span == 0 ? 0 : order_key(T(0x1p29));
}

template <class T>
inline MC<T> to_mc(const ModelCDev& m) {
    MC<T> r;
    r.lambda = (T)m.lambda;
    r.d_thermal = (T)m.d_thermal;
    r.a_bar = (T)m.a_bar;
    r.eps_prime = (T)m.eps_prime;
    r.tol = (T)m.tol;
    r.f_a_bar = (T)m.f_a_bar;
    r.f_eps_prime = (T)m.f_eps_prime;
    r.f_a12 = (T)m.f_a12;
    r.f_tol = (T)m.f_tol;
    r.inv_h2_flux = (T)m.inv_h2_flux;
    r.ih0 = (T)m.inv_h2[0];
    r.ih1 = (T)m.inv_h2[1];
    r.c_far = r.a_bar * r.a_bar;
    r.inv_c_far = T(1) / r.c_far;
    r.quotient_span = quotient_span_of(r);
    // the far forms drop a zero's addition to a face flux, whose sign shows in
    // no result for these parameters
    const bool far = r.quotient_span && r.f_a_bar > T(0.5) && r.d_thermal >= T(0);
    r.far_face = far ? far_below(r.f_tol, false) : 0;
    r.far_center = far ? far_below(r.tol, true) : 0;
    r.safe_below = safe_below_of(r);
    return r;
}

// the division itself, out of line: for operands outside the ranges of the
// shared reciprocal
static __device__ __noinline__ double ieee_quotient(double x, double c) { return x / c; }

// The two ratios of a non-flat face, n1 / c and n2 / c: the IEEE quotients.
// SAFE: the caller knows them to be in range (OpsExact::safe); the tests
// here and the calls behind them cost the FP64 step 7 %.
template <bool SAFE, class T>
__device__ __forceinline__ void ratios(const MC<T>&, float n1, float n2, float c, float& q1, float& q2) {
    q1 = n1 / c;
    q2 = n2 / c;
}
template <bool SAFE, class T>
__device__ __forceinline__ void ratios(const MC<T>& m, double n1, double n2, double c, double& q1, double& q2) {
    if (SAFE || (recip_range(c, m.quotient_span) && fabs(n2) >= kQuotientLow)) {
        const double y = recip_rn(c);
        q1 = quotient_rn(n1, c, y);
        q2 = quotient_rn(n2, c, y);
    } else {
        q1 = ieee_quotient(n1, c);
        q2 = ieee_quotient(n2, c);
    }
}
template <bool SAFE, class T>
__device__ __forceinline__ float ratio(const MC<T>&, float n, float c) { return n / c; }
template <bool SAFE, class T>
__device__ __forceinline__ double ratio(const MC<T>& m, double n, double c) {
    return SAFE || recip_range(c, m.quotient_span) ? quotient_rn(n, c, recip_rn(c)) : ieee_quotient(n, c);
}

// KarmaRappelFlux::face (finite_volume.rs:129-142); its two quotients share
// one reciprocal
template <bool SAFE = false, class T>
__device__ __forceinline__ void kr_face(const MC<T>& m, T dx, T dy, T& a, T& da) {
    T dx2 = dx * dx;
    T dy2 = dy * dy;
    T sum = dx2 + dy2;
    T mag2 = sum * sum;
    if (mag2 <= m.f_tol) {
        a = m.f_a_bar;
        da = T(0);
    } else {
        T q1, q2;
        ratios<SAFE>(m, m.f_eps_prime * (dx2 * dx2 + dy2 * dy2), -(m.f_a12) * dx * dy * (dx2 - dy2), mag2, q1, q2);
        a = m.f_a_bar * (T(1) + q1);
        da = q2;
    }
}

// ModelC::center_anisotropy (phasefield.rs:159-175) from the half
// differences dx = 0.5 (p(i+1) - p(i-1)), dy likewise.
template <bool SAFE = false, class T>
__device__ __forceinline__ T center_anisotropy(const MC<T>& m, T dx, T dy) {
    T dx2 = dx * dx;
    T dy2 = dy * dy;
    T sum = dx2 + dy2;
    T mag2 = sum * sum;
    if (mag2 <= m.tol) return m.a_bar;
    return m.a_bar * (T(1) + ratio<SAFE>(m, m.eps_prime * (dx2 * dx2 + dy2 * dy2), mag2));
}

__device__ __forceinline__ double fma_t(double a, double b, double c) { return fma(a, b, c); }
__device__ __forceinline__ float fma_t(float a, float b, float c) { return fmaf(a, b, c); }

__device__ __forceinline__ double normal_t(uint64_t key, double) { return standard_normal(key); }

// The mobility quotient x / c of a cell, c = a^2 and y = RN(1 / c)
__device__ __forceinline__ double mobility(const MC<double>& m, double x, double c, double y) {
    const double k = quotient_rn(x, c, y);
    return quotient_suspect(x, k, x, k) | (m.quotient_span == 0) ? ieee_quotient(x, c) : k;
}
// of two cells, which share a test (the tests for tiny numerators cost 10080^2
// 0.6 % and 512^2 0.8 %); `divide`: their divisors may be out of range
__device__ __forceinline__ void mobility2(double x0, double c0, double y0, double x1, double c1, double y1, bool divide,
                                          double& k0, double& k1) {
    k0 = quotient_rn(x0, c0, y0);
    k1 = quotient_rn(x1, c1, y1);
    if (divide | quotient_suspect(x0, k0, x1, k1)) {
        k0 = ieee_quotient(x0, c0);
        k1 = ieee_quotient(x1, c1);
    }
}
__device__ __forceinline__ double mobility_recip(double c) { return recip_rn(c); }
__device__ __forceinline__ float mobility(const MC<float>&, float x, float c, float) { return x / c; }
__device__ __forceinline__ void mobility2(float x0, float c0, float, float x1, float c1, float, bool, float& k0,
                                          float& k1) {
    k0 = x0 / c0;
    k1 = x1 / c1;
}
__device__ __forceinline__ float mobility_recip(float) { return 0.0f; }
__device__ __forceinline__ float normal_t(uint64_t key, float) { return standard_normal_f32(key); }

// The exact FP64 arithmetic policy of the step kernels: face fluxes from
// the normal difference dn and the transverse quarter sum 0.25 ((d1 + c) - e)
// (finite_volume.rs:258-283), the cell update (phasefield.rs:395-421) and
// the Euler-Maruyama axpy (driver.rs:210-236), in the reference's operand
// order.
template <class T>
struct OpsExact {
    using Params = MC<T>;
    static constexpr bool kGuarded = true;   // SAFE forms leave a range test out

    // x face: KarmaRappelFlux::face(derx, dery) and j = a (a derx - da dery)
    template <bool SAFE = false>
    static __device__ __forceinline__ T xface(const MC<T>& m, T dn, T d1, T c, T e) {
        const T dt = T(0.25) * (d1 + c - e);
        T a, da;
        kr_face<SAFE>(m, dn, dt, a, da);
        return a * (a * dn - da * dt);
    }
    // y face: face(derx, dery) with derx transverse, j = a (a dery + da derx)
    template <bool SAFE = false>
    static __device__ __forceinline__ T yface(const MC<T>& m, T dn, T d1, T c, T e) {
        const T dt = T(0.25) * (d1 + c - e);
        T a, da;
        kr_face<SAFE>(m, dt, dn, a, da);
        return a * (a * dn + da * dt);
    }
    // The far-field forms: the face fluxes and the cell update with the
    // anisotropy branches decided (kr_face and center_anisotropy both flat):
    // a = f_a_bar, da = 0, and a dn -+ 0 dt is a dn (the transverse difference
    // is finite where the test holds).  The test is conservative (far_below):
    // a pass that fails it takes the general path, whose branches decide each
    // face in the reference's rounding.
    static __device__ __forceinline__ T quarter(T d1, T c, T e) { return T(0.25) * (d1 + c - e); }
    static __device__ __forceinline__ bool far(const MC<T>& m, unsigned faces, unsigned centers) {
        return (faces < m.far_face) & (centers < m.far_center);
    }
    // the SAFE forms leave out the second ratio's own test: where a cell's
    // phase is at least 2^-500 its differences to its neighbours are zero (as
    // the ratio then is) or at least 2^-553, beside which a ratio below 2^-860
    // is lost
    static __device__ __forceinline__ bool safe(const MC<T>& m, unsigned faces, unsigned centers, T p0, T p1) {
        return (max(faces, centers) < m.safe_below) & (min(high_word(p0) << 1, high_word(p1) << 1) >= 2 * 0x20b00000u);
    }
    static __device__ __forceinline__ bool divides(const MC<T>& m) { return m.quotient_span == 0; }
    // of a face's differences, and of a centre's whole ones (p(i+1) - p(i-1))
    static __device__ __forceinline__ unsigned key(T dx, T dy) { return order_key(fma_t(dx, dx, dy * dy)); }
    static __device__ __forceinline__ T xface_far(const MC<T>& m, T dn) { return m.f_a_bar * (m.f_a_bar * dn); }
    static __device__ __forceinline__ T yface_far(const MC<T>& m, T dn) { return m.f_a_bar * (m.f_a_bar * dn); }

    // A cell's dphi/dt = num / c and du/dt = fma(lap, d_thermal, 0.5 dphi/dt),
    // the quotient left open so that the two cells of a pass share its test
    struct Cell {
        T num, c, y, lap;
    };
    // divided outright: a reciprocal of NaN makes the quotient suspect
    static __device__ __forceinline__ void divide(Cell& o) { o.y = T(__longlong_as_double(0x7ff8000000000000LL)); }
    static __device__ __forceinline__ void open(const MC<T>& m, T jr, T jl, T jt, T jb, T p, T uc, T ul, T ur, T up,
                                                T um, Cell& o) {
        const T flux = (jr - jl + jt - jb) * m.inv_h2_flux;
        const T g_prime = fma_t(p * p, p, -p);
        const T one_m_p2 = fma_t(p, -p, T(1));
        const T p_prime = one_m_p2 * one_m_p2;
        o.num = fma_t(m.lambda * uc, -p_prime, flux - g_prime);
        T acc = T(0);
        acc += ((ur - (uc + uc)) + ul) * m.ih0;
        acc += ((up - (uc + uc)) + um) * m.ih1;
        o.lap = acc;
    }
    static __device__ __forceinline__ Cell cell_far(const MC<T>& m, T jr, T jl, T jt, T jb, T p, T uc, T ul, T ur,
                                                    T up, T um) {
        Cell o;
        open(m, jr, jl, jt, jb, p, uc, ul, ur, up, um, o);
        o.c = m.c_far;
        o.y = m.inv_c_far;
        return o;
    }
    template <bool SAFE = false>
    static __device__ __forceinline__ Cell cell_open(const MC<T>& m, T jr, T jl, T jt, T jb, T p, T cdx, T cdy, T uc,
                                                     T ul, T ur, T up, T um) {
        Cell o;
        open(m, jr, jl, jt, jb, p, uc, ul, ur, up, um, o);
        const T a = center_anisotropy<SAFE>(m, T(0.5) * cdx, T(0.5) * cdy);
        o.c = a * a;
        o.y = mobility_recip(o.c);
        return o;
    }
    static __device__ __forceinline__ void close(const MC<T>& m, const Cell& o, T& kphi, T& ku) {
        kphi = mobility(m, o.num, o.c, o.y);
        ku = fma_t(o.lap, m.d_thermal, T(0.5) * kphi);
    }
    // `divide`: see mobility2
    static __device__ __forceinline__ void close2(const MC<T>& m, const Cell& o0, const Cell& o1, bool divide, T& kphi0,
                                                  T& ku0, T& kphi1, T& ku1) {
        mobility2(o0.num, o0.c, o0.y, o1.num, o1.c, o1.y, divide, kphi0, kphi1);
        ku0 = fma_t(o0.lap, m.d_thermal, T(0.5) * kphi0);
        ku1 = fma_t(o1.lap, m.d_thermal, T(0.5) * kphi1);
    }
    static __device__ __forceinline__ void cell(const MC<T>& m, T jr, T jl, T jt, T jb, T p, T cdx, T cdy, T uc,
                                                T ul, T ur, T up, T um, T& kphi, T& ku) {
        close(m, cell_open(m, jr, jl, jt, jb, p, cdx, cdy, uc, ul, ur, up, um), kphi, ku);
    }
    // Multi-grain faces and cell (finite_volume.rs:196-234, phasefield.rs:
    // 378-392): a face's anisotropy in the crystal frame (c0, s0) = (cos, sin)
    // theta0 of the cell being updated, the flux in the lab frame; the centre
    // anisotropy rotated likewise with the flux's constants
    // (center_anisotropy_rotated).  derx/dery are the face's lab-frame
    // differences in the reference's operand order.
    static __device__ __forceinline__ T oxface(const MC<T>& m, T c0, T s0, T derx, T dery) {
        T a, da;
        kr_face(m, c0 * derx + s0 * dery, c0 * dery - s0 * derx, a, da);
        return a * (a * derx - da * dery);
    }
    static __device__ __forceinline__ T oyface(const MC<T>& m, T c0, T s0, T derx, T dery) {
        T a, da;
        kr_face(m, c0 * derx + s0 * dery, c0 * dery - s0 * derx, a, da);
        return a * (a * dery + da * derx);
    }
    static __device__ __forceinline__ Cell ocell_open(const MC<T>& m, T jr, T jl, T jt, T jb, T p, T cdx, T cdy, T c0,
                                                      T s0, T uc, T ul, T ur, T up, T um) {
        Cell o;
        open(m, jr, jl, jt, jb, p, uc, ul, ur, up, um, o);
        const T dx = T(0.5) * cdx, dy = T(0.5) * cdy;
        T a, da;
        kr_face(m, c0 * dx + s0 * dy, c0 * dy - s0 * dx, a, da);
        o.c = a * a;
        o.y = mobility_recip(o.c);
        return o;
    }
    static __device__ __forceinline__ void ocell(const MC<T>& m, T jr, T jl, T jt, T jb, T p, T cdx, T cdy, T c0, T s0,
                                                 T uc, T ul, T ur, T up, T um, T& kphi, T& ku) {
        close(m, ocell_open(m, jr, jl, jt, jb, p, cdx, cdy, c0, s0, uc, ul, ur, up, um), kphi, ku);
    }
    static __device__ __forceinline__ T axpy(T dt, T k, T x) { return x + dt * k; }
    static __device__ __forceinline__ T noise(uint64_t key) { return normal_t(key, T(0)); }
    static __device__ __forceinline__ T add_noise(T x, T scale_amp, T n) { return x + scale_amp * n; }
};

__device__ __forceinline__ int64_t slab_base(const SlabLayout& L, int b, int field) {
    return ((int64_t)b * L.nfields + field) * L.slab_stride;
}

// The eight neighbours of one block of a 2-D Cartesian grid, for ghost
// pushes: face neighbours from the topology table, diagonals by chaining
// (x step, then y step).  -1 where the step leaves the domain through a
// physical boundary; such steps are never taken (mirror images stay in the
// block itself).
struct Nbr2 {
    int b, l, r, d, u, dl, dr, ul, ur;

    __device__ __forceinline__ void load(const CartTopo& topo, int blk) {
        b = blk;
        l = topo.nbr[(blk * 3 + 0) * 2 + 0];
        r = topo.nbr[(blk * 3 + 0) * 2 + 1];
        d = topo.nbr[(blk * 3 + 1) * 2 + 0];
        u = topo.nbr[(blk * 3 + 1) * 2 + 1];
        dl = l >= 0 ? topo.nbr[(l * 3 + 1) * 2 + 0] : -1;
        ul = l >= 0 ? topo.nbr[(l * 3 + 1) * 2 + 1] : -1;
        dr = r >= 0 ? topo.nbr[(r * 3 + 1) * 2 + 0] : -1;
        ur = r >= 0 ? topo.nbr[(r * 3 + 1) * 2 + 1] : -1;
    }
    __device__ __forceinline__ int at(int sx, int sy) const {
        if (sy == 0) return sx == 0 ? b : (sx < 0 ? l : r);
        if (sx == 0) return sy < 0 ? d : u;
        if (sy < 0) return sx < 0 ? dl : dr;
        return sx < 0 ? ul : ur;
    }
};

// Ghost push of 2-D, ghost-width-1 fields: the value of interior cell (i, j)
// goes to every ghost entry whose source it is (the separable map of the
// reference's dimension sweep, cartesian.rs:439-526).  Scalars only, no
// local arrays.
template <class T>
__device__ __forceinline__ void push_ghosts_2d_g1(T* __restrict__ out, const SlabLayout& L, int field,
                                                  const Nbr2& nb, int n0, int n1, int i, int j, T v) {
    const bool lo_x = i == 0, hi_x = i == n0 - 1, lo_y = j == 0, hi_y = j == n1 - 1;
    if (!(lo_x | hi_x | lo_y | hi_y)) return;
    const int sy = L.gdim[0];
    const int sA = nb.l >= 0 ? -1 : 0, iA = nb.l >= 0 ? n0 : -1;
    const int sB = nb.r >= 0 ? 1 : 0, iB = nb.r >= 0 ? -1 : n0;
    const int sC = nb.d >= 0 ? -1 : 0, jC = nb.d >= 0 ? n1 : -1;
    const int sD = nb.u >= 0 ? 1 : 0, jD = nb.u >= 0 ? -1 : n1;
    auto put = [&](int sx, int syy, int ii, int jj) {
        out[slab_base(L, nb.at(sx, syy), field) + (ii + 1) + (int64_t)(jj + 1) * sy] = v;
    };
    if (lo_x) put(sA, 0, iA, j);
    if (hi_x) put(sB, 0, iB, j);
    if (lo_y) put(0, sC, i, jC);
    if (hi_y) put(0, sD, i, jD);
    if (lo_x && lo_y) put(sA, sC, iA, jC);
    if (lo_x && hi_y) put(sA, sD, iA, jD);
    if (hi_x && lo_y) put(sB, sC, iB, jC);
    if (hi_x && hi_y) put(sB, sD, iB, jD);
}

}  // namespace lg
