// Time-integrated BGK-NS interface flux (weno/src/GKMflux.cpp:11-215), FP64
// path.
//
// The reference contracts 1-D moment tables of all three velocity components
// for each of its three Maxwellians (left, right, equilibrium): 41 calls of
// MCal (GKMflux.cpp:225-275) per interface.  Here every Maxwellian is taken in
// its own frame, c = (u, v, w) - U, in which it is an isotropic Gaussian of
// variance s = 1/(2 lambda), and three things follow.
//
// * Slopes.  With b'' the slope of the conserved moments seen from that frame,
//   slopesolver (GKMflux.cpp:280-296) is diagonal but for the energy:
//     h  = a4/2 = kA lambda^2 (b4'' - (K+3) s b0 / 2),   a_i = 2 lambda b_i'',
//     a0 = b0 - (K+3) s h           (kA = 4/(K+3) times the 1/Pr factor, :289).
// * Full-space moments are closed forms, so no full-space table is built:
//     <psi'' (a psi'')>    = (a0 + (K+3) s h, s a_i, (K+3) s (a0 + (K+5) s h) / 2)
//     <psi'' c0 (a psi'')> = (s a1, s (a0 + (K+5) s h), 0, 0, (K+5) s^2 a1 / 2)
//   and the time derivative A of a Maxwellian from its three slopes x, y, z
//   (GKMflux.cpp:128-144) is
//     -A'' = U . a'' + (s D - (K+3) s E, v_x, v_y, v_z; E),
//     D = x1 + y2 + z3,  v_d = d0 + (K+5) s h_d,
//     E = (pr - 1) (U . h) + pr D / (K+3)   (in units of h, as h above).
// * Half-space moments need the table X_n = <u^n> over u > 0 or u < 0 only.
//   For a polynomial sum_i C_i u^i + c1 (...) + c2 (...) in u with transverse
//   weights, N_k = sum_i C_i X_{k+i} gives the density moment, N_{k+1} the
//   normal momentum and (N_{k+2} + (K+2) s N_k + ...) / 2 the energy, so
//   neighbouring moments share the N.  All weights a side contributes to B_
//   (GKMflux.cpp:172-176) and to the flux (GKMflux.cpp:209-212) are collected
//   into one such polynomial each.
//   On u > 0 the equilibrium has the normal slope xl, on u < 0 xr: its moments
//   are those of xr over the full space plus those of xl - xr over u > 0.
// The equilibrium's zeroth-order part of B_, gm1 rho <psi> + gm3 W0
// (GKMflux.cpp:174-178), vanishes identically (gm3 = -gm1 and <psi> rho = W0).
//
// The algebra is the reference's; only the order of evaluation differs, so
// results agree with it to rounding.
//
// Bound: the FP64 pipe.  1097 FP64 instructions per interface (1471 with
// tables of the full space as well and a moment vector per slope); a sweep of
// 256^3 takes 1.543 ms (2.2 ms).
#pragma once

#include "gks_device.cuh"

namespace gks {

// One Maxwellian: state, frame and derived constants.
struct Gauss {
    double den, rinv, U0, U1, U2;
    double p, s;     // pressure, variance 1 / (2 lambda)
    double tl;       // 2 lambda
    double kh;       // kA lambda^2
    double k3, k5;   // (K+3) s, (K+5) s
    double x, e2, g; // sqrt(lambda) U0, exp(-x^2), exp(-x^2) / (2 sqrt(pi lambda))
};

// From the conserved state.  The pressure, whose rounding is most of the error of
// a slow flow's momentum, is taken with as few roundings as there are: one of
// rho E - rho U^2 / 2 and one of its product with gamma - 1 (the kinetic part is
// the smaller one), and goes into the flux as it is.  2 lambda = 1/s and
// sqrt(lambda) are products of one reciprocal square root y of s = p / rho.
// Error of the momenta after a step against 64-bit mantissas, rms relative to
// their largest value, geometric mean over 13 fields of 16^3 to 64^3: 3.9e-17; with p
// and 1/rho as products of 1 / (rho sqrt(rho2p(W))) 7.0e-17; with full-space tables
// and the zeroth-order part of B_ 5.5e-17.
__device__ __forceinline__ Gauss gauss(const double W[5], const FluxConst64 &c)
{
    Gauss m;
    m.den = W[0];
    m.rinv = rcp_cubic(W[0]);
    m.U0 = W[1] * m.rinv;
    m.U1 = W[2] * m.rinv;
    m.U2 = W[3] * m.rinv;
    m.p = c.gm1 * fma(-0.5, fma(W[1], m.U0, fma(W[2], m.U1, W[3] * m.U2)), W[4]);
    m.s = m.p * m.rinv;
    const double y = rsqrt_cubic(m.s);
    m.tl = y * y;
    m.kh = (c.kA4 * m.tl) * m.tl;
    m.k3 = c.K3 * m.s;
    m.k5 = c.K5 * m.s;
    m.x = (0.7071067811865476 * y) * m.U0;
    m.e2 = exp(-m.x * m.x);
    m.g = (0.3989422804014327 * (m.s * y)) * m.e2;
    return m;
}

// X[0..6] = <u^n> over u > 0 (h0 = 0.5 erfc(-x), g > 0) or u < 0 (h0 = 0.5 erfc(x),
// g < 0), and sX[0..3] = s X[0..3] (GKMflux.cpp:52-60).
__device__ __forceinline__ void half_moments(double U, double s, double h0, double g, double X[7], double sX[4])
{
    X[0] = h0;
    X[1] = fma(U, h0, g);
    sX[0] = s * X[0];
    X[2] = fma(U, X[1], sX[0]);
    sX[1] = s * X[1];
    X[3] = fma(2.0, sX[1], U * X[2]);
    sX[2] = s * X[2];
    X[4] = fma(3.0, sX[2], U * X[3]);
    sX[3] = s * X[3];
    X[5] = fma(4.0, sX[3], U * X[4]);
    X[6] = fma(5.0 * s, X[4], U * X[5]);
}

// Conserved-moment vector from the lab into the frame of m, hU = |U|^2 / 2.
__device__ __forceinline__ void to_frame(double b[5], const Gauss &m, double hU)
{
    b[1] = fma(-m.U0, b[0], b[1]);
    b[2] = fma(-m.U1, b[0], b[2]);
    b[3] = fma(-m.U2, b[0], b[3]);
    b[4] = fma(-m.U0, b[1], fma(-m.U1, b[2], fma(-m.U2, b[3], fma(-hU, b[0], b[4]))));
}

// Slope coefficients (a0, a1, a2, a3, h) of sc b'', with tl and kh scaled by sc.
__device__ __forceinline__ void solve(const double b[5], double k3, double sc, double tl, double kh, double a[5])
{
    a[4] = kh * fma(-0.5 * k3, b[0], b[4]);
    a[3] = tl * b[3];
    a[2] = tl * b[2];
    a[1] = tl * b[1];
    a[0] = fma(-k3, a[4], sc * b[0]);
}

// Coefficients in powers of c0 -> in powers of u = U0 + c0.
__device__ __forceinline__ void to_u(double a[5], double U0)
{
    const double t = fma(-a[4], U0, a[1]);
    a[0] = fma(-U0, t, a[0]);
    a[1] = fma(-a[4], U0, t);
}

// One side's pass (SIDE 0: left state over u > 0, 1: right state over u < 0):
// its share of W0 (GKMflux.cpp:71-75), of the transverse right-hand sides by_,
// bz_ of the equilibrium (:109-117), of B_ (:172-176) and of the flux
// (:209-212), put into the sums of `src`.
template <int SIDE, typename Src>
__device__ __forceinline__ void flux_side(const Src &src, const FluxConst64 &c)
{
    double W[5];
    src.template state<SIDE>(W);
    const Gauss m = gauss(W, c);
    const double s = m.s, U0 = m.U0, U1 = m.U1, U2 = m.U2;
    double X[7], sX[4];
    {
        double hp, hm; // 0.5 erfc(+-x)
        half_erfc_pm(m.x, m.e2, hp, hm);
        half_moments(U0, s, SIDE ? hp : hm, SIDE ? -m.g : m.g, X, sX);
    }
    const double r2 = c.K2 * s;            // <rho^2>, rho^2 = c1^2 + c2^2 + xi^2
    const double s2 = s * s;
    const double qq = c.K22 * s2;          // <rho^4> - <rho^2>^2 = 2 (K+2) s^2
    const double k4 = c.K4 * s;
    const double hu = fma(U1, U1, U2 * U2);
    const double c4 = 0.5 * (r2 + hu);
    {
        const double d0 = m.den * X[0];
        src.template sum<SIDE>(Src::kW0 + 0, m.den, X[0]);
        src.template sum<SIDE>(Src::kW0 + 1, m.den, X[1]);
        src.template sum<SIDE>(Src::kW0 + 2, U1, d0);
        src.template sum<SIDE>(Src::kW0 + 3, U2, d0);
        src.template sum<SIDE>(Src::kW0 + 4, c4, d0);
        src.template sum<1>(Src::kW0 + 4, 0.5 * m.den, X[2]);
    }
    const double hU = 0.5 * fma(U0, U0, hu);
    double ax[5], ayz[5], vx, vy, vz, Dt, e0, e1, e2, f0, f1, f2;
    {
        double b[5];
        src.template slope<SIDE, 0>(W, b);
        to_frame(b, m, hU);
        const double sc = c.ksn * m.rinv;
        solve(b, m.k3, sc, sc * m.tl, sc * m.kh, ax);
        vx = fma(m.k5, ax[4], ax[0]);
        to_u(ax, U0);
    }
    const double sc = c.kst * m.rinv, tl = sc * m.tl, kh = sc * m.kh;
    // half-space density, momentum and energy of one transverse slope, lab frame
    auto transverse = [&](int slot, const double a[5]) {
        const double al = fma(a[4], r2, a[0]);
        const double N0 = fma(al, X[0], fma(a[1], X[1], a[4] * X[2]));
        const double N1 = fma(al, X[1], fma(a[1], X[2], a[4] * X[3]));
        const double N2 = fma(al, X[2], fma(a[1], X[3], a[4] * X[4]));
        const double M2 = a[2] * sX[0], M3 = a[3] * sX[0];
        src.template sum<SIDE>(slot + 0, N0);
        src.template sum<SIDE>(slot + 1, N1);
        src.template sum<SIDE>(slot + 2, fma(U1, N0, M2));
        src.template sum<SIDE>(slot + 3, fma(U2, N0, M3));
        src.template sum<SIDE>(slot + 4, fma(0.5, fma(a[4] * qq, X[0], N2), fma(c4, N0, fma(U1, M2, U2 * M3))));
    };
    {
        double a[5], b[5];
        src.template slope<SIDE, 1>(W, b);
        to_frame(b, m, hU);
        solve(b, m.k3, sc, tl, kh, a);
        vy = fma(m.k5, a[4], a[0]);
        Dt = a[2];
        to_u(a, U0);
        transverse(Src::kBy, a);
        e0 = fma(k4, a[4], a[0]);
        e1 = a[1];
        e2 = a[4];
#pragma unroll
        for (int q = 0; q < 5; ++q) ayz[q] = U1 * a[q];
    }
    {
        double a[5], b[5];
        src.template slope<SIDE, 2>(W, b);
        to_frame(b, m, hU);
        solve(b, m.k3, sc, tl, kh, a);
        vz = fma(m.k5, a[4], a[0]);
        Dt += a[3];
        to_u(a, U0);
        transverse(Src::kBz, a);
        f0 = fma(k4, a[4], a[0]);
        f1 = a[1];
        f2 = a[4];
#pragma unroll
        for (int q = 0; q < 5; ++q) ayz[q] = fma(U2, a[q], ayz[q]);
    }
    // -A of this Maxwellian, in powers of u
    double An[5];
    {
        const double D = Dt + fma(2.0 * ax[4], U0, ax[1]); // x1 in powers of c0
        const double E = fma(c.prm1, fma(U0, ax[4], ayz[4]), c.kA4 * D);
        double v[5] = {fma(s, D, -m.k3 * E), vx, vy, vz, E};
        to_u(v, U0);
#pragma unroll
        for (int q = 0; q < 5; ++q) An[q] = fma(U0, ax[q], ayz[q] + v[q]);
    }
    // the convective weight u (x psi) + c1 (y psi) + c2 (z psi) + (U1 y + U2 z) psi
    // by powers of u: C0 .. C3 for the density moments, e (c1) and f (c2) for the
    // transverse momenta over s, Q0, Q1 the excess of the energy over (K+2) s N
    const double C0 = fma(s, Dt, fma(ayz[4], r2, ayz[0]));
    const double C1 = fma(ax[4], r2, ax[0]) + ayz[1];
    const double C2 = ax[1] + ayz[4], C3 = ax[4];
    e0 += ayz[2];
    e1 += ax[2];
    f0 += ayz[3];
    f1 += ax[3];
    const double Q0 = fma(ayz[4], qq, (2.0 * s2) * Dt), Q1 = ax[4] * qq;
    const double aln = fma(An[4], r2, An[0]), qn = An[4] * qq;
    // <psi u^k (wP P + wA (-A) + w1)> for k = K0, lab frame, P the convective weight
    auto collect = [&](int slot, auto K0, double wP, double wA, double w1) {
        constexpr int k = decltype(K0)::value;
        const double D0 = fma(wP, C0, fma(wA, aln, w1));
        const double D1 = fma(wP, C1, wA * An[1]);
        const double D2 = fma(wP, C2, wA * An[4]);
        const double D3 = wP * C3;
        const double N0 = fma(D0, X[k], fma(D1, X[k + 1], fma(D2, X[k + 2], D3 * X[k + 3])));
        const double N1 = fma(D0, X[k + 1], fma(D1, X[k + 2], fma(D2, X[k + 3], D3 * X[k + 4])));
        const double N2 = fma(D0, X[k + 2], fma(D1, X[k + 3], fma(D2, X[k + 4], D3 * X[k + 5])));
        const double M2 = fma(fma(wP, e0, wA * An[2]), sX[k], wP * fma(e1, sX[k + 1], e2 * sX[k + 2]));
        const double M3 = fma(fma(wP, f0, wA * An[3]), sX[k], wP * fma(f1, sX[k + 1], f2 * sX[k + 2]));
        const double R = fma(fma(wP, Q0, wA * qn), X[k], fma(wP * Q1, X[k + 1], N2));
        src.template sum<SIDE>(slot + 0, N0);
        src.template sum<SIDE>(slot + 1, N1);
        src.template sum<SIDE>(slot + 2, fma(U1, N0, M2));
        src.template sum<SIDE>(slot + 3, fma(U2, N0, M3));
        src.template sum<SIDE>(slot + 4, fma(0.5, R, fma(c4, N0, fma(U1, M2, U2 * M3))));
    };
    // gamma weights (GKMflux.cpp:155-157) and time integrals (GKMflux.cpp:186-190)
    const double tau = src.get(Src::kTau), ex = src.get(Src::kTau + 1), igm0 = src.get(Src::kTau + 2);
    const double Pt = tau * (1.0 - ex), tP = tau * Pt;
    const double g5 = Pt * igm0; // tau gm3
    collect(Src::kB, std::integral_constant<int, 0>(), m.den * fma(fma(c.dt, ex, -Pt), igm0, g5), -m.den * g5, 0.0);
    // p3 = P, p4 = -Q - tau P = tau dt ex - 2 tau P, p5 = -tau P
    collect(Src::kF, std::integral_constant<int, 1>(), m.den * fma(tau, c.dt * ex, -2.0 * tP), m.den * tP, m.den * Pt);
}

// The flux.  `src` supplies the inputs when they are needed and keeps the sums
// of the two side passes:
//   src.state<side>(W)        reconstructed state, left (0) or right (1)
//   src.slope<side, d>(W, b)  its differences along d = normal, 1st, 2nd transverse
//   src.cells(WL, WR)         the cell averages either side of the interface
//   src.sum<side>(slot, v)    side 0 stores, side 1 adds; src.get(slot), src.put(slot, v)
// mu/p at the left cell = tau_n / tau_d.  Output F[5], integrated over [0, dt].
// ahead() is called when the inputs have been read (their slots are free).
template <typename Src, typename Ahead>
__device__ __forceinline__ void gks_flux64(const Src &src, double tau_n, double tau_d, const FluxConst64 &c,
                                           const Ahead &ahead, double F[5])
{
    const double dt = c.dt;
    {
        // collision time with the pressure-jump term (GKMflux.cpp:149-150):
        // rho/lambda = 2p, so w = |p_l - p_r| / (p_l + p_r); with
        // p = (gamma - 1) A / rho, A = rho2p(W), multiplied through by
        // rho_l rho_r / (gamma - 1): w = |A_l rho_r - A_r rho_l| / (A_l rho_r + A_r rho_l)
        double W[5];
        src.template state<0>(W);
        const double Al = rho2p(W), rl = W[0];
        src.template state<1>(W);
        const double a = Al * W[0], b = rho2p(W) * rl;
        // tau = tau_n / tau_d + dt w = N / D; one reciprocal r = 1 / (N D) gives
        // tau = N (N r) and 1 / tau = D (D r)
        const double D = tau_d * (a + b);
        const double N = fma(tau_n, a + b, dt * fabs(a - b) * tau_d);
        const double r = rcp_cubic(N * D);
        const double tau = N * (N * r);
        const double ex = exp(-dt * (D * (D * r)));
        src.put(Src::kTau, tau);
        src.put(Src::kTau + 1, ex);
        src.put(Src::kTau + 2, rcp_cubic(fma(-tau, 1.0 - ex, dt))); // 1 / gm0
    }
    flux_side<0>(src, c);
    asm volatile("" ::: "memory"); // one side's state in registers at a time
    flux_side<1>(src, c);
    asm volatile("" ::: "memory");

    // equilibrium state at the interface (GKMflux.cpp:75-98)
    double We[5];
#pragma unroll
    for (int q = 0; q < 5; ++q) We[q] = src.get(Src::kW0 + q);
    const Gauss m = gauss(We, c);
    const double s = m.s, U0 = m.U0, U1 = m.U1, U2 = m.U2;
    const double hu = fma(U1, U1, U2 * U2), hU = 0.5 * fma(U0, U0, hu);
    // slopes (GKMflux.cpp:109-117, 136-137): x on u < 0, its jump xd on u > 0
    double x[5], xd[5], y[5], z[5];
    {
        double b[5], d[5], WL[5], WR[5];
        src.cells(WL, WR);
#pragma unroll
        for (int q = 0; q < 5; ++q) {
            b[q] = WR[q] - We[q];
            d[q] = (We[q] - WL[q]) - b[q];
        }
        const double sc = c.ksn * m.rinv, tl = sc * m.tl, kh = sc * m.kh;
        to_frame(b, m, hU);
        solve(b, m.k3, sc, tl, kh, x);
        to_frame(d, m, hU);
        solve(d, m.k3, sc, tl, kh, xd);
        to_u(xd, U0);
#pragma unroll
        for (int q = 0; q < 5; ++q) b[q] = src.get(Src::kBy + q);
        to_frame(b, m, hU);
        solve(b, m.k3, 1.0, m.tl, m.kh, y);
#pragma unroll
        for (int q = 0; q < 5; ++q) b[q] = src.get(Src::kBz + q);
        to_frame(b, m, hU);
        solve(b, m.k3, 1.0, m.tl, m.kh, z);
    }
    ahead();
    const double vx = fma(m.k5, x[4], x[0]), vy = fma(m.k5, y[4], y[0]), vz = fma(m.k5, z[4], z[0]);
    const double D = x[1] + (y[2] + z[3]);
    // full-space second-order part of the flux, <psi'' u (c . slopes)>, in units of s
    const double G0 = fma(U0, D, vx);
    const double G1 = fma(U0, vx, s * fma(2.0, x[1], D));
    const double G2 = fma(U0, vy, s * (x[2] + y[1]));
    const double G3 = fma(U0, vz, s * (x[3] + z[1]));
    const double G4 = (0.5 * m.k5) * fma(U0, D, fma(fma(2.0, s, m.k5), x[4], x[0]));
    double Ua[5]; // U . slopes
#pragma unroll
    for (int q = 0; q < 5; ++q) Ua[q] = fma(U0, x[q], fma(U1, y[q], U2 * z[q]));
    // half-space moments of the jump of the normal slope, k = 1 (h1) and k = 2 (h2),
    // normal velocity u, transverse c
    double h1[5], h2[5];
    {
        double hp, hm, X[7], sX[4];
        half_erfc_pm(m.x, m.e2, hp, hm);
        half_moments(U0, s, hm, m.g, X, sX);
        const double r2 = c.K2 * s, hq = (c.K22 * (s * s)) * xd[4];
        const double al = fma(xd[4], r2, xd[0]);
        const double N1 = fma(al, X[1], fma(xd[1], X[2], xd[4] * X[3]));
        const double N2 = fma(al, X[2], fma(xd[1], X[3], xd[4] * X[4]));
        const double N3 = fma(al, X[3], fma(xd[1], X[4], xd[4] * X[5]));
        const double N4 = fma(al, X[4], fma(xd[1], X[5], xd[4] * X[6]));
        h1[0] = N1;
        h1[1] = N2;
        h1[2] = xd[2] * sX[1];
        h1[3] = xd[3] * sX[1];
        h1[4] = 0.5 * fma(r2, N1, fma(hq, X[1], N3));
        h2[0] = N2;
        h2[1] = N3;
        h2[2] = xd[2] * sX[2];
        h2[3] = xd[3] * sX[2];
        h2[4] = 0.5 * fma(r2, N2, fma(hq, X[2], N4));
    }
    // A_ (phase III, GKMflux.cpp:159-180): its right-hand side in the frame
    const double tau = src.get(Src::kTau), ex = src.get(Src::kTau + 1), igm0 = src.get(Src::kTau + 2);
    const double Pt = tau * (1.0 - ex);
    double A[5];
    {
        double b[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) b[q] = src.get(Src::kB + q);
        to_frame(b, m, hU);
        const double gm2 = fma(-dt, ex, fma(2.0, Pt, -dt)) * igm0;
        const double sD = s * D;
        const double t1 = fma(-U0, h1[0], h1[1]);
        const double T0 = (fma(m.k3, Ua[4], Ua[0]) + sD) + h1[0];
        const double T1 = fma(s, Ua[1] + vx, t1);
        const double T2 = fma(s, Ua[2] + vy, h1[2]);
        const double T3 = fma(s, Ua[3] + vz, h1[3]);
        const double T4 = fma(0.5, fma(m.k3, fma(m.k5, Ua[4], Ua[0]), m.k5 * sD),
                              fma(-U0, fma(0.5 * U0, h1[0], t1), h1[4]));
        b[0] = fma(gm2, T0, m.rinv * b[0]);
        b[1] = fma(gm2, T1, m.rinv * b[1]);
        b[2] = fma(gm2, T2, m.rinv * b[2]);
        b[3] = fma(gm2, T3, m.rinv * b[3]);
        b[4] = fma(gm2, T4, m.rinv * b[4]);
        solve(b, m.k3, 1.0, m.tl, m.kh, A);
    }
    // flux (GKMflux.cpp:192-213)
    {
        const double p0 = dt - Pt;
        const double p1 = fma(0.5 * dt, dt, -tau * p0);
        const double p2 = fma(-tau, p0, tau * fma(-dt, ex, Pt));
        double a[5];
#pragma unroll
        for (int q = 0; q < 5; ++q) a[q] = fma(p1, A[q], p2 * Ua[q]);
        const double p2s = p2 * s;
        const double m1 = s * a[1], w = fma(m.k5, a[4], a[0]);
        const double f0 = fma(p2s, G0, fma(U0, fma(m.k3, a[4], a[0]), m1));
        const double f1 = fma(p2s, G1, fma(U0, m1, s * w));
        const double f2 = fma(p2s, G2, (U0 * s) * a[2]);
        const double f3 = fma(p2s, G3, (U0 * s) * a[3]);
        const double f4 = fma(p2s, G4, fma(U0, (0.5 * m.k3) * w, (0.5 * m.k5) * m1));
        // frame -> u in the normal direction, plus the half-space part, -> lab
        const double g0 = fma(p2, h2[0], f0);
        const double g1 = fma(p2, h2[1], fma(U0, f0, f1));
        const double g2 = fma(p2, h2[2], f2);
        const double g3 = fma(p2, h2[3], f3);
        const double g4 = fma(p2, h2[4], fma(U0, fma(0.5 * U0, f0, f1), f4));
        const double w0 = p0 * U0;
        F[0] = fma(w0, We[0], fma(m.den, g0, src.get(Src::kF + 0)));
        F[1] = fma(p0, m.p, fma(w0, We[1], fma(m.den, g1, src.get(Src::kF + 1))));
        F[2] = fma(w0, We[2], fma(m.den, fma(U1, g0, g2), src.get(Src::kF + 2)));
        F[3] = fma(w0, We[3], fma(m.den, fma(U2, g0, g3), src.get(Src::kF + 3)));
        F[4] = fma(w0, We[4] + m.p, fma(m.den, fma(U1, g2, fma(U2, g3, fma(0.5 * hu, g0, g4))), src.get(Src::kF + 4)));
    }
}

} // namespace gks
