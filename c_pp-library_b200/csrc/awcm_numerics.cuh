// Device numerics of the AWCM compressible-Euler path: ideal-gas relations, physical fluxes,
// Roe-averaged characteristic projection, WENO-Z / WENO5 reconstruction and the Lax-Friedrichs
// split face flux.  Every expression keeps the reference's operation order (doseongju/C_pp-library),
// and the library is compiled with --fmad=false, so each result is bit-identical to the
// reference's IEEE double arithmetic: division and square root are the correctly rounded ones.
#pragma once
#include <cstdint>

namespace awcm {

constexpr int kGhost = 3;  // ghost width of every field (FIELD_UNIFORM_1D/2D ghost_width 3)

// 11/6, -7/6, 1/3, 5/6, -1/6, 13/12 correctly rounded (the reference builds them as 11.0/6.0, ...).
constexpr double kC11_6 = 0x1.d555555555555p+0;
constexpr double kCm7_6 = -0x1.2aaaaaaaaaaabp+0;
constexpr double kC1_3 = 0x1.5555555555555p-2;
constexpr double kC5_6 = 0x1.aaaaaaaaaaaabp-1;
constexpr double kCm1_6 = -0x1.5555555555555p-3;
constexpr double kC13_12 = 0x1.1555555555555p+0;
// Coarse-level derivative weights of AWCM_1D/AWCM_2D (Wavelet/AWCM_1D.h:21, 36-39).
constexpr double kD1 = 0x1.5555555555555p-1;    // 2/3
constexpr double kD2 = -0x1.5555555555555p-4;   // -1/12
constexpr double kD01 = -0x1.5555555555555p-2;  // -1/3
constexpr double kD11 = -0.5;
constexpr double kD21 = 1.0;
constexpr double kD31 = -0x1.5555555555555p-3;  // -1/6
constexpr double kD02 = 0x1.5555555555555p-4;   // 1/12
constexpr double kD12 = -0x1.5555555555555p-1;  // -2/3
constexpr double kD22 = 0.0;
constexpr double kD32 = 0x1.5555555555555p-1;   // 2/3

enum Scheme : int { kWenoZ = 0, kWeno5 = 1, kScalarAdvection = 2 };  // 2: the 1D scalar path only

__device__ __forceinline__ double sqr(double x) { return x * x; }
__device__ __forceinline__ double absd(double x) { return x < 0 ? -x : x; }
__device__ __forceinline__ double maxd(double a, double b) { return a > b ? a : b; }

// ---------------------------------------------------------------------------------- divisions
// About 70 (1D) and 113 (2D) divisions make up most of a face flux.  The compiler's IEEE division is
// a branch to a special-case path away from a plain instruction sequence, so two of them never
// overlap: 114 cycles each on a lone warp, 25 cycles a warp where many share the FP64 pipe.  Most
// of a face's divisors divide several values (a cell's density, twice the Roe speed of sound, a
// reconstruction's weight sum), so the divisor's reciprocal is computed once, and a quotient takes
// five multiply-adds without a branch (29 cycles on a lone warp, 17 a warp where many share the pipe).
//
// Both are correctly rounded, i.e. the same bits as the IEEE division.  This is Markstein's method
// (P. W. Markstein, Computation of elementary functions on the IBM RISC System/6000 processor, 1990;
// Muller et al., Handbook of Floating-Point Arithmetic, division with an FMA): a reciprocal within
// one ulp becomes RN(1/b) by one more Newton step, unless b's significand is all ones; and with y =
// RN(1/b) and q within one ulp of a/b, RN(q + (a - b q) y) is RN(a/b), a - b q being exact.
// It holds as long as no step under- or overflows, so a policy object collects whether an operand
// left the safe range (`bad`), and the caller then evaluates the whole expression again with
// IEEE divisions.

// IEEE division.
struct IeeeDiv {
    typedef double Divisor;
    static constexpr bool checked = false;
    __device__ __forceinline__ double by(double b) { return b; }
    __device__ __forceinline__ double twice(double b) { return 2 * b; }
    __device__ __forceinline__ double quot(double a, double b) { return a / b; }
    __device__ __forceinline__ double quot_pos(double a, double b) { return a / b; }
    __device__ __forceinline__ double recip(double b) { return 1.0 / b; }
    __device__ __forceinline__ void range(double, int, int) {}
    __device__ __forceinline__ void range_or_0(double, int, int) {}
};
// Division by shared reciprocals.
struct SharedDiv {
    struct Divisor {
        double b, y;
    };
    static constexpr bool checked = true;
    bool bad = false;
    // |x| in [2^lo, 2^hi), or zero (range_or_0); NaN and infinities are outside.
    __device__ __forceinline__ void range(double x, int lo, int hi)
    {
        const unsigned e = ((unsigned)__double2hiint(x) & 0x7fffffffu) - ((unsigned)(lo + 1023) << 20);
        bad |= e >= ((unsigned)(hi - lo) << 20);
    }
    __device__ __forceinline__ void range_or_0(double x, int lo, int hi)
    {
        const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
        bad |= (h | (unsigned)__double2loint(x)) != 0u &&
               h - ((unsigned)(lo + 1023) << 20) >= ((unsigned)(hi - lo) << 20);
    }
    // b normal, within [2^-900, 2^900]
    __device__ __forceinline__ Divisor by(double b)
    {
        double y;
        asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(b));  // relative error 2^-20 (measured over all of them)
        const double e = fma(-b, y, 1.0);
        y = fma(y, fma(e, e, e), y);     // 2^-60 before rounding: within one ulp
        y = fma(y, fma(-b, y, 1.0), y);  // RN(1/b), or for the all-ones significand 2^-k instead of 2^-k (1 + 2^-52)
        const unsigned lo = (unsigned)__double2loint(b);
        const bool ones = (((unsigned)__double2hiint(b) | 0xfff00000u) & lo) == 0xffffffffu;
        return Divisor{b, __hiloint2double(__double2hiint(y), __double2loint(y) | (ones ? 1 : 0))};
    }
    __device__ __forceinline__ double recip(double b) { return by(b).y; }
    // The divisor 2 b from that of b.
    __device__ __forceinline__ Divisor twice(const Divisor& d) { return Divisor{2 * d.b, 0.5 * d.y}; }
    // a > 0, or any a where the sign of a zero quotient does not matter
    __device__ __forceinline__ double quot_pos(double a, const Divisor& d)
    {
        double q = a * d.y;
        q = fma(fma(-d.b, q, a), d.y, q);
        return fma(fma(-d.b, q, a), d.y, q);
    }
    __device__ __forceinline__ double quot(double a, const Divisor& d)
    {
        const double q0 = a * d.y;
        double q = fma(fma(-d.b, q0, a), d.y, q0);
        q = fma(fma(-d.b, q, a), d.y, q);
        // a = -0 keeps its sign
        return (((unsigned)__double2hiint(a) & 0x7fffffffu) | (unsigned)__double2loint(a)) ? q : q0;
    }
};
// The safe range of a point's and a face's operands: the density in [2^-20, 2^20), momenta and energies 0 or
// in [2^-100, 2^30), the Roe speed of sound in [2^-20, 2^30), the LF speed below 2^60.  Whatever is divided
// or divides is then 0 or within [2^-640, 2^710]: the largest are a reconstruction's weights (a
// characteristic value is below 2^281, its smoothness below 2^569, tau / (b + 1e-40) below 2^702), the
// smallest a difference of products of u, f and c.  A reconstruction's tau may be smaller, where 1 + tau / d
// is 1 whatever the quotient's last bits are.
constexpr int kSafeLo = -100, kSafeHi = 30, kSafeRho = 20, kSafeC = -20, kSafeAlpha = 60;

// WENOZ5::ReconstructLeft (WENOZ.h:75-104): tau = |b0 - b2|, alpha_k = d_k (1 + tau/(b_k + eps)),
// eps = 1e-40.  WENO5::ReconstructLeft (WENO.h:71-99): alpha_k = d_k / (eps + b_k)^2, eps = 1e-6.
// wz_eps: WENOZ5::eps (WENOZ.h:13-18), a public member of the reference solver, 1e-40 by default.
// wz_delta > 0 replaces tau = |b0 - b2| by sqrt((b0 - b2)^2 + wz_delta^2) (the differentiable
// mode of the gradient checks; the reference has only |.|).
template <int SCHEME, class DV>
__device__ __forceinline__ double recon_left(DV& dv, double ll, double l, double c, double r, double rr,
                                             double wz_eps = 1e-40, double wz_delta = 0.0)
{
    const double b0 = kC13_12 * sqr(c - 2 * r + rr) + 0.25 * sqr(3 * c - 4 * r + rr);
    const double b1 = kC13_12 * sqr(l - 2 * c + r) + 0.25 * sqr(l - r);
    const double b2 = kC13_12 * sqr(ll - 2 * l + c) + 0.25 * sqr(ll - 4 * l + 3 * c);
    double w0, w1, w2;
    if (SCHEME == kWeno5) {
        const double eps = 1e-6;
        const double e0 = sqr(eps + b0), e1 = sqr(eps + b1), e2 = sqr(eps + b2);
        dv.range(e0, -60, 700), dv.range(e1, -60, 700), dv.range(e2, -60, 700);
        const double a0 = dv.quot_pos(0.1, dv.by(e0));
        const double a1 = dv.quot_pos(0.6, dv.by(e1));
        const double a2 = dv.quot_pos(0.3, dv.by(e2));
        const auto s = dv.by(a0 + a1 + a2);
        w0 = dv.quot_pos(a0, s), w1 = dv.quot_pos(a1, s), w2 = dv.quot_pos(a2, s);
    } else {
        const double eps = wz_eps;
        const double tau = wz_delta > 0 ? sqrt(sqr(b0 - b2) + sqr(wz_delta)) : absd(b0 - b2);
        const double d0 = b0 + eps, d1 = b1 + eps, d2 = b2 + eps;
        if (tau == 0 && d0 > 0 && d1 > 0 && d2 > 0) {
            // tau / d_k is a signed zero and 1 + (+-0) = 1, so alpha_k = d_k exactly; their sum
            // 0.1 + 0.6 + 0.3 rounds to exactly 1.0 in IEEE double, so the normalised weights are
            // the d_k themselves.  All six divisions are skipped (a zero quotient sends IEEE
            // division down its slow path, and piecewise-constant stencils make tau = 0 common).
            w0 = 0.1, w1 = 0.6, w2 = 0.3;
        } else {
            const double a0 = 0.1 * (1 + dv.quot_pos(tau, dv.by(d0)));
            const double a1 = 0.6 * (1 + dv.quot_pos(tau, dv.by(d1)));
            const double a2 = 0.3 * (1 + dv.quot_pos(tau, dv.by(d2)));
            const auto s = dv.by(a0 + a1 + a2);
            w0 = dv.quot_pos(a0, s), w1 = dv.quot_pos(a1, s), w2 = dv.quot_pos(a2, s);
        }
    }
    double left = w0 * (kC11_6 * c + kCm7_6 * r + kC1_3 * rr);
    left += w1 * (kC1_3 * l + kC5_6 * c + kCm1_6 * r);
    left += w2 * (kCm1_6 * ll + kC5_6 * l + kC1_3 * c);
    return left;
}

template <int SCHEME>
__device__ __forceinline__ double recon_left(double ll, double l, double c, double r, double rr)
{
    IeeeDiv dv;
    return recon_left<SCHEME>(dv, ll, l, c, r, rr);
}

// ------------------------------------------------------------------------------------ 1D gas
// IDEAL_GAS_1D (IDEAL_GAS_EQUATIONS.h:8-58), EULER_EQUATION_1D::ComputeFu (EULER_EQUATION.h:16-26).
__device__ __forceinline__ double pressure1(double q0, double q1, double q2, double g)
{
    return (g - 1) * (q2 - 0.5 * sqr(q1) / q0);
}
__device__ __forceinline__ double sound1(double q0, double q1, double q2, double g)
{
    return sqrt(g * pressure1(q0, q1, q2, g) / q0);
}
template <class DV>
__device__ __forceinline__ double pressure1(DV& dv, double q1, double q2, const typename DV::Divisor& rho, double g)
{
    return (g - 1) * (q2 - dv.quot(0.5 * sqr(q1), rho));
}
// |u| + c (EULER_EQUATION.h:42-47).
template <class DV>
__device__ __forceinline__ double speed1(DV& dv, double q0, double q1, double q2, double g)
{
    dv.range(q0, -kSafeRho, kSafeRho);
    dv.range_or_0(q1, kSafeLo, kSafeHi);
    const auto rho = dv.by(q0);
    const double gp = g * pressure1(dv, q1, q2, rho, g);
    dv.range_or_0(gp, kSafeLo, 3 * kSafeHi);
    const double u = dv.quot(q1, rho);
    return absd(u) + sqrt(dv.quot(gp, rho));
}
template <class DV>
__device__ __forceinline__ void flux1(DV& dv, const double* q, double g, double* f)
{
    dv.range(q[0], -kSafeRho, kSafeRho);
    dv.range_or_0(q[1], kSafeLo, kSafeHi);
    const auto r = dv.by(q[0]);
    const double rho = q[0], u = dv.quot(q[1], r), E = q[2], p = pressure1(dv, q[1], q[2], r, g);
    f[0] = rho * u;
    f[1] = rho * u * u + p;
    f[2] = (E + p) * u;
}

// ROE_SOLVER_1D::Inversion (ROESOLVER.h:27-36), with 0.4/(c*c) precomputed as kc (same value) and
// c2 the divisor 2 c.
template <class DV>
__device__ __forceinline__ void inv1(DV& dv, double u, double H, double c, double kc, const typename DV::Divisor& c2,
                                     const double* b, double* x)
{
    double x2 = (H - u * u) * b[0] + u * b[1] - b[2];
    x2 *= kc;
    double x3 = b[1] + (c - u) * b[0] - c * x2;
    x3 = dv.quot(x3, c2);
    x[0] = b[0] - x2 - x3;
    x[1] = x2;
    x[2] = x3;
}

// WENOZ_EULER_SOLVER_1D::ComputeFlux (WENOZ.h:160-205) / WENO_EULER_SOLVER_1D::ComputeFlux
// (WENO.h:129-174).  s[p] are the six cells -3..+2 of the face, alpha the LF speed.
template <int SCHEME, class DV>
__device__ __forceinline__ void face_flux_1d(DV& dv, const double (&s)[6][3], double alpha, double g, double* out)
{
    // the cells' velocities and pressures (EULER_EQUATION_1D::ComputeFu) and the Roe average of the two
    // cells at the face (ROE_SOLVER_1D::RoeAverage) share the divisions by the densities
    double f[6][3], uc[2], Hc[2];
    dv.range(alpha, kSafeLo, kSafeAlpha);
#pragma unroll
    for (int p = 0; p < 6; ++p) {
        const double* q = s[p];
        dv.range(q[0], -kSafeRho, kSafeRho);
        dv.range_or_0(q[1], kSafeLo, kSafeHi);
        dv.range_or_0(q[2], kSafeLo, kSafeHi);
        const auto rho = dv.by(q[0]);
        const double u = dv.quot(q[1], rho), pr = pressure1(dv, q[1], q[2], rho, g);
        f[p][0] = q[0] * u;
        f[p][1] = q[0] * u * u + pr;
        f[p][2] = (q[2] + pr) * u;
        if (p == 2 || p == 3) {
            uc[p - 2] = u;
            Hc[p - 2] = dv.quot(q[2] + pr, rho);
        }
    }
    const double sl = sqrt(s[2][0]), sr = sqrt(s[3][0]);
    const auto den = dv.by(sl + sr);
    const double u = dv.quot(sl * uc[0] + sr * uc[1], den);
    const double H = dv.quot(sl * Hc[0] + sr * Hc[1], den);
    const double c = sqrt((g - 1) * (H - 0.5 * u * u));
    dv.range(c, kSafeC, kSafeHi);
    const double kc = dv.quot_pos(0.4, dv.by(c * c));
    const auto c2 = dv.by(2 * c);
    double fp[6][3], fm[6][3];
#pragma unroll
    for (int p = 0; p < 6; ++p) {
        double RQ[3], RF[3];
        inv1(dv, u, H, c, kc, c2, s[p], RQ);
        inv1(dv, u, H, c, kc, c2, f[p], RF);
#pragma unroll
        for (int k = 0; k < 3; ++k) {
            fp[p][k] = 0.5 * (RF[k] + alpha * RQ[k]);
            fm[p][k] = 0.5 * (RF[k] - alpha * RQ[k]);
        }
    }
    double S[3];
#pragma unroll
    for (int k = 0; k < 3; ++k) {
        const double lr = recon_left<SCHEME>(dv, fp[4][k], fp[3][k], fp[2][k], fp[1][k], fp[0][k]);
        const double rl = recon_left<SCHEME>(dv, fm[1][k], fm[2][k], fm[3][k], fm[4][k], fm[5][k]);
        S[k] = lr + rl;
    }
    const double r1[3] = {1, u - c, H - u * c};
    const double r2[3] = {1, u, 0.5 * (u * u)};
    const double r3[3] = {1, u + c, H + u * c};
#pragma unroll
    for (int k = 0; k < 3; ++k) out[k] = S[0] * r1[k] + S[1] * r2[k] + S[2] * r3[k];
}

// ------------------------------------------------------------------------------------ 2D gas
// IDEAL_GAS_2D (IDEAL_GAS_EQUATIONS.h:60-111), EULER_EQUATION_2D (EULER_EQUATION.h:64-156).
__device__ __forceinline__ double pressure2(double q0, double q1, double q2, double q3, double g)
{
    return (g - 1) * (q3 - 0.5 * (sqr(q1) + sqr(q2)) / q0);
}
__device__ __forceinline__ double sound2(const double* q, double g)
{
    return sqrt(g * pressure2(q[0], q[1], q[2], q[3], g) / q[0]);
}
// DIR 0: ComputeFu (F), DIR 1: ComputeGu (G).
template <int DIR>
__device__ __forceinline__ void flux2(const double* q, double g, double* f)
{
    const double rho = q[0], u = q[1] / q[0], v = q[2] / q[0], E = q[3];
    const double p = pressure2(q[0], q[1], q[2], q[3], g);
    if (DIR == 0) {
        f[0] = rho * u;
        f[1] = rho * u * u + p;
        f[2] = rho * v * u;
        f[3] = (E + p) * u;
    } else {
        f[0] = rho * v;
        f[1] = rho * u * v;
        f[2] = rho * v * v + p;
        f[3] = (E + p) * v;
    }
}

// |u| + c and |v| + c of a point (EULER_EQUATION.h:118-142).
template <class DV>
__device__ __forceinline__ void speeds2(DV& dv, const double* q, double g, double& sx, double& sy)
{
    dv.range(q[0], -kSafeRho, kSafeRho);
    dv.range_or_0(q[1], kSafeLo, kSafeHi);
    dv.range_or_0(q[2], kSafeLo, kSafeHi);
    const auto rho = dv.by(q[0]);
    const double gp = g * ((g - 1) * (q[3] - dv.quot(0.5 * (sqr(q[1]) + sqr(q[2])), rho)));
    dv.range_or_0(gp, kSafeLo, 3 * kSafeHi);
    const double c = sqrt(dv.quot(gp, rho));
    sx = absd(dv.quot(q[1], rho)) + c;
    sy = absd(dv.quot(q[2], rho)) + c;
}

// ROE_SOLVER_2D::Inversion_X (ROESOLVER.h:73-84; Inversion_Y with the momenta exchanged); kc = 0.4 / c / c, same
// value, c2 the divisor 2 c, A = H - u * u - v * v.
template <class DV>
__device__ __forceinline__ void inv2(DV& dv, double A, double u, double v, double c, double kc,
                                     const typename DV::Divisor& c2, const double* b, double* x)
{
    double x3 = A * b[0] + u * b[1] + v * b[2] - b[3];
    x3 *= kc;
    const double x2 = b[2] - v * b[0];
    double x4 = b[1] + (c - u) * b[0] - c * x3;
    x4 = dv.quot(x4, c2);
    x[0] = b[0] - x3 - x4;
    x[1] = x2;
    x[2] = x3;
    x[3] = x4;
}

// The x flux of one cell (flux2<0>) with its velocities and total enthalpy from one reciprocal.
template <class DV>
__device__ __forceinline__ void cell_flux2(DV& dv, const double* q, double g, double* f, double* prim)
{
    dv.range(q[0], -kSafeRho, kSafeRho);
    dv.range_or_0(q[1], kSafeLo, kSafeHi);
    dv.range_or_0(q[2], kSafeLo, kSafeHi);
    dv.range_or_0(q[3], kSafeLo, kSafeHi);
    const auto r = dv.by(q[0]);
    const double rho = q[0], u = dv.quot(q[1], r), v = dv.quot(q[2], r), E = q[3];
    const double p = (g - 1) * (q[3] - dv.quot(0.5 * (sqr(q[1]) + sqr(q[2])), r));
    f[0] = rho * u;
    f[1] = rho * u * u + p;
    f[2] = rho * v * u;
    f[3] = (E + p) * u;
    if (prim) {
        prim[0] = u;
        prim[1] = v;
        prim[2] = dv.quot(E + p, r);
    }
}

// WENOZ_EULER_SOLVER_2D::ComputeFluxX / ComputeFluxY, WENOZ.h:236-320, with the Roe average of the two
// cells at the face (ROE_SOLVER_2D::RoeAverage, ROESOLVER.h:49-70).  s[p] = cells -3..+2 across the face.
// One code for both directions: a y face passes its cells, and gets its flux, with the momenta exchanged.
// ComputeFluxY then takes the same operations on the same operands, but for the order in which the Roe
// velocities' squares are subtracted from H.
// false, with nothing in out, where the cells, alpha or the speed of sound are outside the range of DV: a state in
// units that are out of range everywhere then pays for little more than the IEEE divisions (scaled by 2^25, a
// 2049 x 2049 step takes 860 us; 991 with both ways in full, 949 with IEEE divisions alone).
template <class DV>
__device__ __forceinline__ bool face_flux_2d(DV& dv, const double (&s)[6][4], bool y, double alpha, double g, double* out,
                                             double wz_eps = 1e-40, double wz_delta = 0.0)
{
    double f[6][4], L[3], R[3];
    dv.range(alpha, kSafeLo, kSafeAlpha);
#pragma unroll
    for (int p = 0; p < 6; ++p) cell_flux2(dv, s[p], g, f[p], p == 2 ? L : p == 3 ? R : nullptr);
    const double sl = sqrt(s[2][0]), sr = sqrt(s[3][0]);
    const auto den = dv.by(sl + sr);
    const double u = dv.quot(sl * L[0] + sr * R[0], den);
    const double v = dv.quot(sl * L[1] + sr * R[1], den);
    const double H = dv.quot(sl * L[2] + sr * R[2], den);
    const double c = sqrt(0.4 * (H - 0.5 * (u * u + v * v)));
    dv.range(c, kSafeC, kSafeHi);
    if constexpr (DV::checked)
        if (dv.bad) return false;
    const auto c1 = dv.by(c);
    const double kc = dv.quot_pos(dv.quot_pos(0.4, c1), c1);
    const auto c2 = dv.twice(c1);
    const double uu = u * u, vv = v * v;
    const double A = y ? (H - vv) - uu : (H - uu) - vv;
    double fp[6][4], fm[6][4];
#pragma unroll
    for (int p = 0; p < 6; ++p) {
        double RQ[4], RF[4];
        inv2(dv, A, u, v, c, kc, c2, s[p], RQ);
        inv2(dv, A, u, v, c, kc, c2, f[p], RF);
#pragma unroll
        for (int k = 0; k < 4; ++k) {
            fp[p][k] = 0.5 * (RF[k] + alpha * RQ[k]);
            fm[p][k] = 0.5 * (RF[k] - alpha * RQ[k]);
        }
    }
    double S[4];
#pragma unroll
    for (int k = 0; k < 4; ++k) {
        const double lr = recon_left<kWenoZ>(dv, fp[4][k], fp[3][k], fp[2][k], fp[1][k], fp[0][k], wz_eps, wz_delta);
        const double rl = recon_left<kWenoZ>(dv, fm[1][k], fm[2][k], fm[3][k], fm[4][k], fm[5][k], wz_eps, wz_delta);
        S[k] = lr + rl;
    }
    double r1[4], r2[4], r3[4], r4[4];
    r1[0] = 1, r2[0] = 0, r3[0] = 1, r4[0] = 1;
    r1[1] = u - c, r2[1] = 0, r3[1] = u, r4[1] = u + c;
    r1[2] = v, r2[2] = 1, r3[2] = v, r4[2] = v;
    r1[3] = H - u * c, r2[3] = v, r3[3] = 0.5 * (u * u + v * v), r4[3] = H + u * c;
#pragma unroll
    for (int k = 0; k < 4; ++k) out[k] = S[0] * r1[k] + S[1] * r2[k] + S[2] * r3[k] + S[3] * r4[k];
    return true;
}

}  // namespace awcm
