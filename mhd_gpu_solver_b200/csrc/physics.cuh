// Point-wise GLM-MHD numerics for the sm_100a stage kernels.
//
// Written for this project from the reference's numerical method; each function names the
// reference file:line whose arithmetic it follows, so the FP64 form agrees with the reference CPU
// path to round-off. The operation order is the reference's but for the FP64 fast speed, HLL
// weights, energy and energy flux and both forms' half slopes, which are regrouped where that saves
// operations. Against 80-bit arithmetic the regrouped FP64 form is no further off than the
// reference's order was: over 30 solves of 128 x 128 to 512 x 512 (10 to 200 steps, all limiters,
// masked and non-ideal ones among them) the relative L2 error is 2.37e-16 on average against
// 2.38e-16. All functions are templated on the arithmetic type T (double for the plain form, float
// for the FP32-mixed form).
#pragma once

#include <cstdint>

namespace mhdb {

enum LimiterKind : int { kMinmod = 0, kMC = 1, kVanLeer = 2 };

// Rotated frame: n = face normal, t = in-plane tangential (x-faces: n=x, t=y; y-faces: n=y,
// t=x); include/mhd/kernels/muscl_hll.hpp:11-13,23-31.
template <class T>
struct PrimN {
    T rho, vn, vt, vz, p, bn, bt, bz, psi;
};

template <class T>
struct FluxN {
    T rho, mn, mt, mz, e, bn, bt, bz, psi;
};

// Whether x is zero, negative or too small for the FP64 approximations below (which flush inputs
// under 2^-1022), from its upper word in two integer comparisons beside the FP64 pipe; false for
// NaN, so a select on it passes NaN through.
__device__ __forceinline__ bool vanishes(double x)
{
    const int hi = __double2hiint(x);
    return hi < 0x00100000 && static_cast<unsigned>(hi) <= 0xfff00000u;
}
// Whether x lies in [2^-440, 2^440), by its upper word.
__device__ __forceinline__ bool moderate(double x)
{
    return static_cast<unsigned>(__double2hiint(x)) - 0x24700000u < 0x37000000u;
}

// Reciprocal and square root.
// FP64: the hardware approximation (rcp / rsqrt.approx.ftz.f64; relative error 2^-19.9 measured)
// and one third-order correction (Householder's iteration of order two: with e = 1 - x y the
// reciprocal is y (1 + e + e^2) up to e^3; with e = 1 - x y^2 the reciprocal root is
// y (1 + e/2 + 3 e^2/8) up to e^3). The reciprocal is within 2^-53 (mean 0.38 x 2^-53 over 10^6
// arguments, as the IEEE division), the root and the reciprocal root within 1.5 x 2^-53 (mean 0.38),
// a factor on it adds 2^-53. The FP64 kernels are bound by the FP64 pipe and its latencies; unlike
// the compiler's division and square root these have no branch to a slow path, so the scheduler can
// interleave the chains of a face, and about half the FP64 instructions. With the fast speed's one
// reciprocal root, the limiter's reciprocal per component (below) and integer sign tests, a 4096^2
// van Leer step went from 2.72 to 2.16 ms, a masked non-ideal 2048^2 step from 1.33 to 1.05 ms. For
// operands whose reciprocal is normal too: others take rcp_any and sqrt_any, lose the result in a
// select, or give the NaN that the cell comes to in any case (a density that is zero, subnormal or
// infinite).
// FP32 (the FP32-mixed form): the hardware approximations rcp.approx.ftz / sqrt.approx.ftz (PTX
// ISA; about 1 ulp), used only where the operand is a positive normal number or the result is
// discarded by a select (inverse densities, 1/(sR - sL) with sR - sL >= 2 c_h, |B|, the van
// Leer denominator a + b with ab > 0, and the non-negative fast-speed discriminants).
__device__ __forceinline__ double fast_rcp(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    return fma(y, fma(e, e, e), y);
}
__device__ __forceinline__ float fast_rcp(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
// 1/x of any x: an operand that is zero, infinite or NaN gives what the division gives (the
// approximation has these right, its correction has not), a subnormal one infinity, and one above
// 2^1022 zero.
__device__ __forceinline__ double rcp_any(double x)
{
    double y;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-x, y, 1.0);
    const double r = fma(y, fma(e, e, e), y);
    const bool normal = (static_cast<unsigned>(__double2hiint(x)) << 1) - 0x00200000u < 0xff800000u;
    return normal ? r : y;
}
__device__ __forceinline__ float rcp_any(float x)
{
    return fast_rcp(x);
}
// a / sqrt(x), corrected as a y (1 + e/2 + 3 e^2/8), so that a factor costs nothing extra.
__device__ __forceinline__ double scaled_rsqrt(double a, double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double e = fma(-(x * y), y, 1.0);
    const double t = a * y;
    return fma(t * e, fma(0.375, e, 0.5), t);
}
// sqrt(x) = x / sqrt(x); 0 where x vanishes or is negative.
__device__ __forceinline__ double sqrt_or_zero(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double t = x * y;
    const double e = fma(-t, y, 1.0);
    const double r = fma(t * e, fma(0.375, e, 0.5), t);
    return vanishes(x) ? 0.0 : r;
}
// sqrt(x) of any x >= 0 or NaN: infinity and NaN as they are; a subnormal one counts as zero.
__device__ __forceinline__ double sqrt_any(double x)
{
    const double r = sqrt_or_zero(x);
    return __double2hiint(x) >= 0x7ff00000 ? x : r;
}
__device__ __forceinline__ float fast_sqrt(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float sqrt_any(float x)
{
    return fast_sqrt(x);
}

// mhd::simd scalar min/max (include/mhd/simd.hpp:40-47): the first operand wins ties and
// NaN comparisons, exactly as (b < a) ? b : a.
template <class T>
__device__ __forceinline__ T vmin(T a, T b)
{
    return (b < a) ? b : a;
}
template <class T>
__device__ __forceinline__ T vmax(T a, T b)
{
    return (a < b) ? b : a;
}
// FP32 (the FP32-mixed form): the single-instruction IEEE minNum/maxNum, which agree with the
// reference's selection for every pair of numbers and differ only in which operand a NaN yields.
template <>
__device__ __forceinline__ float vmin<float>(float a, float b)
{
    return fminf(a, b);
}
template <>
__device__ __forceinline__ float vmax<float>(float a, float b)
{
    return fmaxf(a, b);
}

template <class T>
__device__ __forceinline__ T tabs(T a)
{
    return a < T(0) ? -a : a;
}

// include/mhd/kernels/muscl_hll.hpp:33-38
template <class T>
__device__ __forceinline__ T minmod(T a, T b)
{
    return (a * b <= T(0)) ? T(0) : ((fabs(a) < fabs(b)) ? a : b);
}

// Half of the limited slope, lim(a, b) / 2, computed directly (halving is exact, so this is the
// value 0.5 * lim(a, b)): minmod minmod(a/2, b/2) and MC minmod((a + b)/4, minmod(a, b))
// (include/mhd/kernels/muscl_hll.hpp:33-47), van Leer ab / (a + b) where ab > 0, else 0 (van
// Leer's 1974 harmonic limiter 2ab / (a + b); the reference has none,
// include/mhd/mhd_types.hpp:44). FP32 van Leer: ab * rcp(a + b) without a branch; when ab > 0
// after rounding, a and b share their sign and max(|a|, |b|) >= 2^-74.5, so a + b is a normal
// number and the approximate reciprocal is within its stated error; otherwise the select returns
// 0. FP64 van Leer the same with fast_rcp and the sign of ab read from its upper word (flat: zero,
// negative or below 2^-1042; NaN passes; a + b is at least 2^-521 elsewhere): a reciprocal per
// component costs three FP64 instructions and no branch, where inverting a cell's nine sums with
// one division cost 3.5 each, a range test and a fallback (per step: 1024^2 167 -> 162 us, masked
// non-ideal 2048^2 1.09 -> 1.03 ms). FP64 MC: where ab > 0 the central slope has the sign of both,
// so its product test is left out.
template <int L, class T>
__device__ __forceinline__ T limit_half_slope(T a, T b)
{
    if constexpr (L == kMinmod) {
        return minmod(T(0.5) * a, T(0.5) * b);
    } else if constexpr (L == kMC && sizeof(T) == 8) {
        const T m = fabs(a) < fabs(b) ? a : b;
        const T c = T(0.25) * (a + b);
        return (a * b <= T(0)) ? T(0) : (fabs(c) < fabs(m) ? c : m);
    } else if constexpr (L == kMC) {
        return minmod(T(0.25) * (a + b), minmod(a, b));
    } else if constexpr (sizeof(T) == 8) {
        const T p = a * b;
        const int hi = __double2hiint(p);
        const bool flat = hi <= 0 && static_cast<unsigned>(hi) <= 0xfff00000u;
        const T q = p * fast_rcp(a + b);
        return flat ? T(0) : q;
    } else {
        const float p = a * b;
        const float q = p * fast_rcp(a + b);
        return (p <= 0.0f) ? 0.0f : q;
    }
}

// limit_half_slope of nine components (a[c], b[c]).
template <int L, class T>
__device__ __forceinline__ void limit_half_slopes(const T (&a)[9], const T (&b)[9], T (&out)[9])
{
#pragma unroll
    for (int c = 0; c < 9; ++c) {
        out[c] = limit_half_slope<L>(a[c], b[c]);
    }
}

// Fast magnetosonic speed along n in the reference's form, from 1/rho;
// include/mhd/kernels/muscl_hll.hpp:70-87.
template <class T>
__device__ __forceinline__ T reference_fast_speed(const PrimN<T>& W, T inv_rho, T gamma)
{
    const T cs2 = gamma * W.p * inv_rho;
    const T bn2 = W.bn * W.bn;
    const T b2 = bn2 + W.bt * W.bt + W.bz * W.bz;
    const T va2 = b2 * inv_rho;
    const T van2 = bn2 * inv_rho;
    const T sum = cs2 + va2;
    const T disc = vmax(sum * sum - T(4) * cs2 * van2, T(0));
    const T cf2 = T(0.5) * (sum + sqrt_any(disc));
    return sqrt_any(vmax(cf2, T(0)));
}

// The same of an FP64 state whose density and pressure are moderate. The density is factored out:
// with A = gamma p + B^2, c_f = sqrt((A + sqrt(A^2 - 4 gamma p B_n^2)) / (2 rho)) =
// X / sqrt(2 rho X) with X = A + sqrt(...), which needs one reciprocal root in place of a division
// and a root. A^2 and rho X stay normal then: gamma p >= 2^-440, and a B^2 above 2^512 leaves a
// pressure computed from the energy beside it no value between 0 and 2^440 (its steps are 2^-53 of
// the energy). Other states (vanishing and negative densities and pressures, infinities, NaN,
// extreme units) take the reference's form, so that a speed that overflows is infinite here too.
__device__ __forceinline__ double moderate_fast_speed(const PrimN<double>& W, double gamma)
{
    const double gp = gamma * W.p;
    const double bn2 = W.bn * W.bn;
    const double A = gp + (bn2 + W.bt * W.bt + W.bz * W.bz);
    const double X = A + sqrt_or_zero(A * A - (4.0 * gp) * bn2);
    return scaled_rsqrt(X, (W.rho + W.rho) * X);
}

// Fast speeds of a face's FP64 states that are not moderate. They are found in the branch that
// chooses the states and taken by a select: a branch around the speeds, or a general flux beside the
// usual one, splits the face's arithmetic and costs 4 to 10 % of a step, this costs 0 to 3 %.
struct GivenSpeeds {
    bool given = false;
    double left = 0.0, right = 0.0;
};
__device__ __forceinline__ bool moderate_states(const PrimN<double>& L, const PrimN<double>& R)
{
    return moderate(L.rho) && moderate(L.p) && moderate(R.rho) && moderate(R.p);
}

// Conserved state and GLM-MHD flux along n; include/mhd/kernels/muscl_hll.hpp:89-124.
template <class T>
__device__ __forceinline__ void conserved_and_flux(const PrimN<T>& W, T inv_gm1, T ch2,
                                                   FluxN<T>& U, FluxN<T>& F)
{
    const T mn = W.rho * W.vn;
    const T mt = W.rho * W.vt;
    const T mz = W.rho * W.vz;
    const T b2 = W.bn * W.bn + W.bt * W.bt + W.bz * W.bz;
    const T pmag = T(0.5) * b2;
    const T pstar = W.p + pmag;
    const T vb = W.vn * W.bn + W.vt * W.bt + W.vz * W.bz;
    T energy;
    if constexpr (sizeof(T) == 8) { // rho v^2 from the momenta: two FP64 instructions fewer
        energy = W.p * inv_gm1 + T(0.5) * (b2 + (mn * W.vn + mt * W.vt + mz * W.vz));
    } else {
        const T v2 = W.vn * W.vn + W.vt * W.vt + W.vz * W.vz;
        energy = W.p * inv_gm1 + T(0.5) * W.rho * v2 + pmag;
    }

    U.rho = W.rho;
    U.mn = mn;
    U.mt = mt;
    U.mz = mz;
    U.e = energy;
    U.bn = W.bn;
    U.bt = W.bt;
    U.bz = W.bz;
    U.psi = W.psi;

    F.rho = mn;
    F.mn = mn * W.vn + pstar - W.bn * W.bn;
    F.mt = mn * W.vt - W.bn * W.bt;
    F.mz = mn * W.vz - W.bn * W.bz;
    if constexpr (sizeof(T) == 8) {
        F.e = (energy + pstar) * W.vn + W.bn * (W.psi - vb);
    } else {
        F.e = (energy + pstar) * W.vn - W.bn * vb + W.psi * W.bn;
    }
    F.bn = W.psi;
    F.bt = W.vn * W.bt - W.vt * W.bn;
    F.bz = W.vn * W.bz - W.vz * W.bn;
    F.psi = ch2 * W.bn;
}

// HLL flux with Dedner GLM wave-speed bounds (-c_h, +c_h) from the two face states, with the
// upwind and degenerate (|sR - sL| < 1e-14) branches; include/mhd/kernels/muscl_hll.hpp:170-208.
// speeds: the fast speeds of FP64 states that are not moderate.
template <class T>
__device__ __forceinline__ FluxN<T> hll_flux(const PrimN<T>& WL, const PrimN<T>& WR, T gamma,
                                             T inv_gm1, T c_h, const GivenSpeeds& speeds)
{
    T cfL, cfR;
    if constexpr (sizeof(T) == 8) {
        const T fL = moderate_fast_speed(WL, gamma), fR = moderate_fast_speed(WR, gamma);
        cfL = speeds.given ? speeds.left : fL;
        cfR = speeds.given ? speeds.right : fR;
    } else {
        cfL = reference_fast_speed(WL, fast_rcp(WL.rho), gamma);
        cfR = reference_fast_speed(WR, fast_rcp(WR.rho), gamma);
    }
    const T sL = vmin(vmin(WL.vn - cfL, WR.vn - cfR), -c_h);
    const T sR = vmax(vmax(WL.vn + cfL, WR.vn + cfR), c_h);

    const T ch2 = c_h * c_h;
    FluxN<T> UL, UR, FL, FR;
    conserved_and_flux(WL, inv_gm1, ch2, UL, FL);
    conserved_and_flux(WR, inv_gm1, ch2, UR, FR);

    const T denom = sR - sL;
    const T inv_denom = fast_rcp(denom);
    const T sLsR = sL * sR;
    const bool use_left = sL >= T(0);
    const bool use_right = sR <= T(0);
    const bool degenerate = fabs(denom) < T(1.0e-14);

    // The three weights folded into 1/(sR - sL) once per face: four operations per component.
    const T wR = sR * inv_denom, wL = sL * inv_denom, wLR = sLsR * inv_denom;
    auto hll = [&](T fl, T fr, T ul, T ur) { return wR * fl - wL * fr + wLR * (ur - ul); };
    auto combine = [&](T fl, T fr, T ul, T ur) {
        const T mid = degenerate ? T(0.5) * (fl + fr) : hll(fl, fr, ul, ur);
        return use_left ? fl : (use_right ? fr : mid);
    };

    FluxN<T> F;
    if (c_h >= T(1.0e-14)) {
        // sL <= -c_h < 0 < c_h <= sR (or NaN) and sR - sL >= 2 c_h > 1e-14: neither upwind
        // branch nor the degenerate one can be taken, so the selection below returns the HLL
        // average for every component (NaN included). c_h is the same for every face of a
        // launch, so this branch does not diverge.
        F.rho = hll(FL.rho, FR.rho, UL.rho, UR.rho);
        F.mn = hll(FL.mn, FR.mn, UL.mn, UR.mn);
        F.mt = hll(FL.mt, FR.mt, UL.mt, UR.mt);
        F.mz = hll(FL.mz, FR.mz, UL.mz, UR.mz);
        F.e = hll(FL.e, FR.e, UL.e, UR.e);
        F.bn = hll(FL.bn, FR.bn, UL.bn, UR.bn);
        F.bt = hll(FL.bt, FR.bt, UL.bt, UR.bt);
        F.bz = hll(FL.bz, FR.bz, UL.bz, UR.bz);
        F.psi = hll(FL.psi, FR.psi, UL.psi, UR.psi);
        return F;
    }
    F.rho = combine(FL.rho, FR.rho, UL.rho, UR.rho);
    F.mn = combine(FL.mn, FR.mn, UL.mn, UR.mn);
    F.mt = combine(FL.mt, FR.mt, UL.mt, UR.mt);
    F.mz = combine(FL.mz, FR.mz, UL.mz, UR.mz);
    F.e = combine(FL.e, FR.e, UL.e, UR.e);
    F.bn = combine(FL.bn, FR.bn, UL.bn, UR.bn);
    F.bt = combine(FL.bt, FR.bt, UL.bt, UR.bt);
    F.bz = combine(FL.bz, FR.bz, UL.bz, UR.bz);
    F.psi = combine(FL.psi, FR.psi, UL.psi, UR.psi);
    return F;
}

// max(|vx| + cf_x, |vy| + cf_y) from conserved values; include/mhd/kernels/muscl_hll.hpp:211-239.
template <class T>
__device__ __forceinline__ T cell_max_signal_speed(T rho, T mx, T my, T mz, T energy, T bx, T by,
                                                   T bz, T gamma)
{
    const T inv_rho = rcp_any(rho);
    PrimN<T> W;
    W.rho = rho;
    W.vn = mx * inv_rho;
    W.vt = my * inv_rho;
    W.vz = mz * inv_rho;
    const T ekin = T(0.5) * (mx * mx + my * my + mz * mz) * inv_rho;
    const T emag = T(0.5) * (bx * bx + by * by + bz * bz);
    W.p = (gamma - T(1)) * (energy - ekin - emag);
    W.bn = bx;
    W.bt = by;
    W.bz = bz;
    W.psi = T(0);
    PrimN<T> Wy = W;
    Wy.vn = W.vt;
    Wy.vt = W.vn;
    Wy.bn = by;
    Wy.bt = bx;
    T cx, cy;
    if constexpr (sizeof(T) == 8) {
        cx = moderate_fast_speed(W, gamma);
        cy = moderate_fast_speed(Wy, gamma);
        if (__builtin_expect(!(moderate(rho) && moderate(W.p)), 0)) {
            cx = reference_fast_speed(W, inv_rho, gamma);
            cy = reference_fast_speed(Wy, inv_rho, gamma);
        }
    } else {
        cx = reference_fast_speed(W, inv_rho, gamma);
        cy = reference_fast_speed(Wy, inv_rho, gamma);
    }
    const T sx = fabs(W.vn) + cx;
    const T sy = fabs(Wy.vn) + cy;
    return vmax(sx, sy);
}

// Conserved -> primitive as the reference RHS does it (reciprocal of rho, then products);
// include/mhd/kernels/cpu_rows.hpp:129-155. Writes rho, vx, vy, vz, p, bx, by, bz, psi.
template <class T>
__device__ __forceinline__ void cons_to_prim(const T* u, T gm1, T* w)
{
    const T rho = u[0], mx = u[1], my = u[2], mz = u[3], e = u[4];
    const T bx = u[5], by = u[6], bz = u[7];
    const T inv_rho = fast_rcp(rho);
    const T ekin = T(0.5) * (mx * mx + my * my + mz * mz) * inv_rho;
    const T emag = T(0.5) * (bx * bx + by * by + bz * bz);
    w[0] = rho;
    w[1] = mx * inv_rho;
    w[2] = my * inv_rho;
    w[3] = mz * inv_rho;
    w[4] = gm1 * (e - ekin - emag);
    w[5] = bx;
    w[6] = by;
    w[7] = bz;
    w[8] = u[8];
}

// Reflective copy of one fluid neighbour into a solid cell: to_primitive (division form), negate
// the normal velocity, floor rho and p at 1e-12, to_conservative;
// include/mhd/mask.hpp:123-137 with include/mhd/mhd_physics.hpp:23-57. axis 0 = x neighbour.
template <class T>
__device__ __forceinline__ void reflect_fill(const T* s, int axis, T gm1, T* out)
{
    const T rho = s[0], mx = s[1], my = s[2], mz = s[3], E = s[4];
    const T bx = s[5], by = s[6], bz = s[7];
    T vx = mx / rho;
    T vy = my / rho;
    const T vz = mz / rho;
    const T e_kin = T(0.5) * (mx * mx + my * my + mz * mz) / rho;
    const T e_mag = T(0.5) * (bx * bx + by * by + bz * bz);
    T p = gm1 * (E - e_kin - e_mag);
    T r = rho;
    if (axis == 0) {
        vx = -vx;
    } else {
        vy = -vy;
    }
    if (r < T(1e-12)) {
        r = T(1e-12);
    }
    if (p < T(1e-12)) {
        p = T(1e-12);
    }
    const T ek = T(0.5) * r * (vx * vx + vy * vy + vz * vz);
    const T em = T(0.5) * (bx * bx + by * by + bz * bz);
    out[0] = r;
    out[1] = r * vx;
    out[2] = r * vy;
    out[3] = r * vz;
    out[4] = p / gm1 + ek + em;
    out[5] = bx;
    out[6] = by;
    out[7] = bz;
    out[8] = s[8];
}

// Benign state of a solid cell without fluid neighbours: rho = p = 1 at rest, zero B and psi
// (include/mhd/mask.hpp:141-146).
template <class T>
__device__ __forceinline__ void isolated_fill(T gm1, T* out)
{
    out[0] = T(1);
    out[1] = T(0);
    out[2] = T(0);
    out[3] = T(0);
    out[4] = T(1) / gm1; // p / (gamma - 1) + 0 kinetic + 0 magnetic
    out[5] = T(0);
    out[6] = T(0);
    out[7] = T(0);
    out[8] = T(0);
}

// Generalised Ohm's law E = eta_O J + eta_H J x B / |B| + eta_A (J x B) x B / |B|^2, Hall and
// ambipolar skipped where |B|^2 < 1e-14; include/mhd/nonideal.hpp:63-102.
struct NonIdealCoef {
    int ohmic, hall, ambipolar;
    double eta_ohm, eta_hall, eta_ambipolar;
};

template <class T>
__device__ __forceinline__ void nonideal_e(T Jx, T Jy, T Jz, T Bx, T By, T Bz,
                                           const NonIdealCoef& c, T& Ex, T& Ey, T& Ez)
{
    Ex = T(0);
    Ey = T(0);
    Ez = T(0);
    if (c.ohmic) {
        const T eo = T(c.eta_ohm);
        Ex += eo * Jx;
        Ey += eo * Jy;
        Ez += eo * Jz;
    }
    if (!(c.hall || c.ambipolar)) {
        return;
    }
    const T B2 = Bx * Bx + By * By + Bz * Bz;
    if (B2 < T(1.0e-14)) {
        return;
    }
    const T cx = Jy * Bz - Jz * By;
    const T cy = Jz * Bx - Jx * Bz;
    const T cz = Jx * By - Jy * Bx;
    if (c.hall) {
        T invB;
        if constexpr (sizeof(T) == 8) {
            invB = scaled_rsqrt(1.0, B2);
        } else {
            invB = fast_rcp(fast_sqrt(B2));
        }
        const T eh = T(c.eta_hall);
        Ex += eh * cx * invB;
        Ey += eh * cy * invB;
        Ez += eh * cz * invB;
    }
    if (c.ambipolar) {
        const T dx = cy * Bz - cz * By;
        const T dy = cz * Bx - cx * Bz;
        const T dz = cx * By - cy * Bx;
        const T invB2 = fast_rcp(B2);
        const T ea = T(c.eta_ambipolar);
        Ex += ea * dx * invB2;
        Ey += ea * dy * invB2;
        Ez += ea * dz * invB2;
    }
}

} // namespace mhdb
