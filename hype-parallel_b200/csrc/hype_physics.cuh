// hype_physics.cuh -- device-side physics of HyPE-2D's primitive-variable right
// hand side: stiffened-gas systems (Kapila five-equation, Baer-Nunziato, Euler),
// WENO reconstruction, admissibility checks, Rusanov flux + fluctuation.
//
// Bit compatibility: every expression keeps the operand order of the reference
// C it restates (file:line at each function) and the translation units that
// include this header are compiled with --fmad=false, so each product and sum
// rounds on its own exactly as the reference's `gcc -O2` code does on x86-64.
// IEEE division and square root are correctly rounded on both sides.
#pragma once
#include "hype_div.cuh"
#include <cstdint>
#include <utility>
#include <type_traits>

namespace hype {

enum : int { SYS_EULER = 0, SYS_KAPILA = 1, SYS_BN = 2 };
// HyPE-2D/hype.h:76 enum bndry_type
enum : int { BC_WALL = 0, BC_INLET = 1, BC_PERIODIC = 2, BC_REFLECTIVE = 3, BC_TRANSMISSIVE = 4,
             // internal: a y-slab edge inside the grid; its ghost rows are the neighbouring
             // slab's rows, kept in the slab's own halo rows (rows -3..-1 or ny..ny+2)
             BC_HALO = 5 };

// error bits reported through the device error word
enum : unsigned { ERR_INADMISSIBLE_FACE = 1u, ERR_NONFINITE = 2u, ERR_TMA_TIMEOUT = 4u, ERR_BAD_LAUNCH = 8u };

struct EosBase {
    double g1, g2, pi1, pi2;
    int fix_p2;   // Baer-Nunziato: 0 = flux pressure of phase 2 read from V[8] as baer_nunziato.c:271 does
    int cr;       // 1: the constants are within CrDiv's range
    double r_g12, r_g1, r_g2;   // the correctly rounded reciprocals of (g1 - 1)(g2 - 1), g1 - 1, g2 - 1
    __host__ __device__ void reciprocals()
    {
        r_g12 = 1.0 / ((g1 - 1.0) * (g2 - 1.0));
        r_g1 = 1.0 / (g1 - 1.0);
        r_g2 = 1.0 / (g2 - 1.0);
        cr = g1 >= 1.0 + 0x1p-20 && g1 <= 1024.0 && g2 >= 1.0 + 0x1p-20 && g2 <= 1024.0 && pi1 >= 0.0 && pi1 <= 0x1p100 &&
             pi2 >= 0.0 && pi2 <= 0x1p100;
    }
};
struct Eos : EosBase {
    // constants the FP64 performance form (hype_physics_fast.cuh) reads instead of
    // dividing by them; filled by derive() at the start of each of its tiles
    double g1m1, g2m1, inv_g1m1, inv_g2m1, inv_g12, g1pi1, g2pi2, c1, c2;
    __host__ __device__ void derive()
    {
        g1m1 = g1 - 1.0;
        g2m1 = g2 - 1.0;
        inv_g1m1 = 1.0 / g1m1;
        inv_g2m1 = 1.0 / g2m1;
        inv_g12 = 1.0 / (g1m1 * g2m1);
        g1pi1 = g1 * pi1;
        g2pi2 = g2 * pi2;
        c1 = g1pi1 * g2m1;   // alpha_1 gamma_1 pi_1 (gamma_2 - 1) per unit alpha_1 (kapila_5eqn.c:27)
        c2 = g2pi2 * g1m1;
    }
};

// HyPE-2D/hype.h:50-62
constexpr double PRS_FLOOR = 1.0e-12;
constexpr double RHO_FLOOR = 1.0e-14;
constexpr double SMALL_NUM = 1.0e-12;
constexpr double R1_6 = 1. / 6.;
constexpr double R13_3 = 13. / 3.;
constexpr double R7_6 = 7. / 6.;
constexpr double R11_120 = 11. / 120.;
constexpr double R1_12 = 1. / 12.;
constexpr double R41_60 = 41. / 60.;

template <int V> using ic = std::integral_constant<int, V>;
template <class F, int... Is>
__host__ __device__ __forceinline__ void static_for_impl(F &&f, std::integer_sequence<int, Is...>) { (f(ic<Is>{}), ...); }
template <int N, class F>
__host__ __device__ __forceinline__ void static_for(F &&f) { static_for_impl(f, std::make_integer_sequence<int, N>{}); }

// ---------------------------------------------------------------------------
// modal basis (reconstruction.c:11-100) and quadrature tables (hype.c:194-305)
// ---------------------------------------------------------------------------
constexpr double GP = 0.28867513459481287;

constexpr double basis_c(double x, double y, int n)
{
    return n == 0 ? 1.0 : n == 1 ? x : n == 2 ? y : n == 3 ? x * x - 1. / 12. : n == 4 ? y * y - 1. / 12.
         : n == 5 ? x * y : n == 6 ? x * (x * x - 3. / 20.) : n == 7 ? y * (y * y - 3. / 20.)
         : n == 8 ? y * (x * x - 1. / 12.) : n == 9 ? x * (y * y - 1. / 12.) : 0.0;
}
constexpr double basis_gx_c(double x, double y, int n)
{
    return n == 1 ? 1.0 : n == 3 ? 2.0 * x : n == 5 ? y : n == 6 ? 3.0 * x * x - 3. / 20. : n == 8 ? 2.0 * x * y
         : n == 9 ? (y * y - 1. / 12.) : 0.0;
}
constexpr double basis_gy_c(double x, double y, int n)
{
    return n == 2 ? 1.0 : n == 4 ? 2.0 * y : n == 5 ? x : n == 7 ? 3.0 * y * y - 3. / 20. : n == 8 ? (x * x - 1. / 12.)
         : n == 9 ? 2.0 * x * y : 0.0;
}

template <int N>
struct Quad {
    static constexpr int NDOF = (N + 1) * (N + 2) / 2;
    static constexpr int NFGP = N < 2 ? 1 : 2;
    static constexpr int NVGP = N < 2 ? 1 : 4;
    static constexpr int NNODE = 4 * NFGP;
    static constexpr double xf(int q) { return N < 2 ? 0.0 : (q == 0 ? -GP : GP); }
    static constexpr double wf(int q) { return N < 2 ? 1.0 : 0.5; }
    static constexpr double xv(int q) { return N < 2 ? 0.0 : (q < 2 ? -GP : GP); }
    static constexpr double yv(int q) { return N < 2 ? 0.0 : ((q & 1) ? GP : -GP); }
    static constexpr double wv(int q) { return N < 2 ? 1.0 : 0.25; }
    static constexpr double xn(int q)
    {
        return N < 2 ? (q == 0 ? 0.5 : q == 1 ? -0.5 : 0.0)
                     : (q < 2 ? 0.5 : q < 4 ? -0.5 : ((q & 1) ? GP : -GP));
    }
    static constexpr double yn(int q)
    {
        return N < 2 ? (q == 2 ? 0.5 : q == 3 ? -0.5 : 0.0)
                     : (q < 4 ? ((q & 1) ? GP : -GP) : (q < 6 ? 0.5 : -0.5));
    }
    // face f: 0 left (x=-1/2), 1 right, 2 bottom (y=-1/2), 3 top
    static constexpr double face_x(int f, int q) { return f == 0 ? -0.5 : f == 1 ? 0.5 : xf(q); }
    static constexpr double face_y(int f, int q) { return f == 2 ? -0.5 : f == 3 ? 0.5 : xf(q); }
    static constexpr double phi_face(int f, int q, int k) { return basis_c(face_x(f, q), face_y(f, q), k); }
    static constexpr double phi_node(int q, int k) { return basis_c(xn(q), yn(q), k); }
    static constexpr double phi_vol(int q, int k) { return basis_c(xv(q), yv(q), k); }
    static constexpr double dphi_vol_x(int q, int k) { return basis_gx_c(xv(q), yv(q), k); }
    static constexpr double dphi_vol_y(int q, int k) { return basis_gy_c(xv(q), yv(q), k); }
    // gradphiFace_x / _y (hype.c:255-285), d = 0 (x) or 1 (y)
    static constexpr double dphi_face(int f, int q, int d, int k)
    {
        return d == 0 ? basis_gx_c(face_x(f, q), face_y(f, q), k) : basis_gy_c(face_x(f, q), face_y(f, q), k);
    }
};

// Accumulate sum_k c[k]*phi(k) from 0.0 in ascending k, as the reference's
// loops do.  A term with phi == 0 is dropped at compile time: the running sum
// starts at +0 and can never become -0, so adding (c*0) = +-0 never changes it
// for finite c.
template <int NDOF, class PHI>
__device__ __forceinline__ double poly_eval(const double *c, PHI phi)
{
    double v = 0.0;
    static_for<NDOF>([&](auto k) {
        constexpr double p = PHI::template at<decltype(k)::value>();
        if constexpr (p != 0.0) {
            if constexpr (p == 1.0) v = v + c[k];
            else v = v + c[k] * p;
        }
    });
    return v;
}
template <int N, int F, int Q> struct PhiFace { template <int K> static constexpr double at() { return Quad<N>::phi_face(F, Q, K); } };
template <int N, int Q> struct PhiNode { template <int K> static constexpr double at() { return Quad<N>::phi_node(Q, K); } };
template <int N, int Q> struct PhiVol { template <int K> static constexpr double at() { return Quad<N>::phi_vol(Q, K); } };
template <int N, int Q> struct DPhiVolX { template <int K> static constexpr double at() { return Quad<N>::dphi_vol_x(Q, K); } };
template <int N, int Q> struct DPhiVolY { template <int K> static constexpr double at() { return Quad<N>::dphi_vol_y(Q, K); } };

// x in [2^LO, 2^HI), by its high word (one integer subtraction and comparison: the
// FP64 pipe, which bounds the tiles, has no part in it); false for NaN and -x
template <int LO, int HI>
__device__ __forceinline__ bool exp_in(double x)
{
    return (unsigned)__double2hiint(x) - ((unsigned)(1023 + LO) << 20) < ((unsigned)(HI - LO) << 20);
}
// x in [0, 1)
__device__ __forceinline__ bool frac_in(double x) { return (unsigned)__double2hiint(x) < 0x3ff00000u; }

// How a system's functions divide.  IeeeDiv: the compiler's division.  CrDiv: the
// branch-free correctly rounded forms of hype_div.cuh, whose chains interleave; the values
// named to pos(), frac(), mag(), den() and num() bound every operand, and where one is outside
// special() holds and the caller repeats the function with IeeeDiv.
struct IeeeDiv {
    __device__ __forceinline__ double operator()(double a, double b) const { return a / b; }
    __device__ __forceinline__ double by_const(double a, double b, double) const { return a / b; }   // third: 1/b, correctly rounded
    __device__ __forceinline__ double rcp(double) const { return 0.0; }
    __device__ __forceinline__ double quot(double a, double b, double) const { return a / b; }       // third: rcp(b)
    __device__ __forceinline__ void pos(double) const {}
    __device__ __forceinline__ void frac(double) const {}
    __device__ __forceinline__ void num(double) const {}
    __device__ __forceinline__ void mag(double) const {}
    __device__ __forceinline__ void den(double) const {}
};
struct CrDiv {
    bool in = true;
    __device__ __forceinline__ double operator()(double a, double b) const { return div_rn(a, b, rcp_rn(b)); }
    __device__ __forceinline__ double by_const(double a, double b, double rb) const { return div_rn(a, b, rb); }
    __device__ __forceinline__ double rcp(double b) const { return rcp_rn(b); }
    __device__ __forceinline__ double quot(double a, double b, double y) const { return div_rn(a, b, y); }
    __device__ __forceinline__ void pos(double x) { in = in && exp_in<-100, 100>(x); }    // a density, a p + P_inf
    __device__ __forceinline__ void frac(double x) { in = in && exp_in<-100, 0>(x); }     // a volume fraction
    // of any sign: a p + P_inf (negative in the trace gas of a liquid under tension), a divisor that
    // may cancel
    __device__ __forceinline__ void mag(double x) { in = in && exp_in<-100, 100>(fabs(x)); }
    __device__ __forceinline__ void den(double x) { in = in && exp_in<-300, 300>(fabs(x)); }
    __device__ __forceinline__ void num(double x)                                          // a numerator of any sign: 0 or |x| >= 2^-300
    {
        const unsigned h = (unsigned)__double2hiint(x) & 0x7fffffffu;
        in = in && (h - ((1023u - 300u) << 20) < (500u << 20) || (h | (unsigned)__double2loint(x)) == 0u);
    }
    __device__ __forceinline__ bool special() const { return !in; }
};

// ---------------------------------------------------------------------------
// PDE systems (primitive-variable path)
//
// pad_quick<c>(v): value v of variable c lies in a range where, for constants that
// quick_eos accepts, pad() is true whatever the other variables are within theirs.
// Almost every cell is accepted by it, without the sound speeds' divisions; the rest
// takes pad() itself.
// ---------------------------------------------------------------------------
template <int SYS> struct System;

// kapila_5eqn.c: cons [a1 r1, a2 r2, rho u, rho v, E, a1], prim [r1, r2, u, v, p, a1]
template <> struct System<SYS_KAPILA> {
    static constexpr int NV = 6;
    static constexpr int RX0 = 2, RX1 = -1, RY0 = 3, RY1 = -1;   // rhs_function_prim.c:124-125, 253-254
    static constexpr int RXV = 3, RYV = 2;                         // tangential, VISCOUS only: :126-127, :255-256
    // kapila_5eqn.c:14-35
    template <class Dv>
    __device__ __forceinline__ static void cons2prim_dv(const EosBase &e, const double *Q, double *V, Dv &dv)
    {
        double alpha_1 = Q[5];
        double alpha_2 = 1.0 - alpha_1;
        double rho = Q[0] + Q[1];
        dv.frac(alpha_1); dv.pos(rho); dv.num(Q[0]); dv.num(Q[1]); dv.num(Q[2]); dv.num(Q[3]);
        const double ir = dv.rcp(rho);
        double u = dv.quot(Q[2], rho, ir);
        double v = dv.quot(Q[3], rho, ir);
        double E = Q[4];
        double ei = E - 0.5 * rho * (u * u + v * v);
        double G1m1 = e.g1 - 1.0;
        double G2m1 = e.g2 - 1.0;
        const double pn = ei * G1m1 * G2m1 - alpha_1 * e.g1 * e.pi1 * G2m1 - alpha_2 * e.g2 * e.pi2 * G1m1;
        dv.num(pn);
        double p = dv(pn, alpha_1 * G2m1 + alpha_2 * G1m1);
        V[0] = dv(Q[0], alpha_1);
        V[1] = dv(Q[1], alpha_2);
        V[2] = u;
        V[3] = v;
        V[4] = p;
        V[5] = alpha_1;
    }
    __device__ __forceinline__ static void cons2prim(const EosBase &e, const double *Q, double *V)
    {
        IeeeDiv dv;
        cons2prim_dv(e, Q, V, dv);
    }
    // kapila_5eqn.c:41-61
    template <class Dv>
    __device__ __forceinline__ static void prim2cons(const EosBase &e, Dv &dv, const double *V, double *Q)
    {
        double alpha_1 = V[5];
        double alpha_2 = 1.0 - alpha_1;
        double rho = alpha_1 * V[0] + alpha_2 * V[1];
        double u = V[2], v = V[3], p = V[4];
        double G1m1 = e.g1 - 1.0;
        double G2m1 = e.g2 - 1.0;
        double ei = dv.by_const(p * (alpha_1 * G2m1 + alpha_2 * G1m1) + alpha_1 * e.g1 * e.pi1 * G2m1 + alpha_2 * e.g2 * e.pi2 * G1m1, G1m1 * G2m1, e.r_g12);
        double E = ei + 0.5 * rho * (u * u + v * v);
        Q[0] = alpha_1 * V[0];
        Q[1] = alpha_2 * V[1];
        Q[2] = rho * V[2];
        Q[3] = rho * V[3];
        Q[4] = E;
        Q[5] = alpha_1;
    }
    // kapila_5eqn.c:326-371
    template <int DIR, class Dv>
    __device__ __forceinline__ static double flux(const EosBase &e, Dv &dv, const double *V, double *F, bool &bad)
    {
        constexpr double nx = DIR == 0 ? 1.0 : 0.0, ny = DIR == 0 ? 0.0 : 1.0;
        double alpha_1 = V[5];
        double alpha_2 = 1.0 - alpha_1;
        double rho_1 = V[0], rho_2 = V[1];
        double rho = alpha_1 * rho_1 + alpha_2 * rho_2;
        double u = V[2], v = V[3], p = V[4];
        double G1m1 = e.g1 - 1.0;
        double G2m1 = e.g2 - 1.0;
        double ei = dv.by_const(p * (alpha_1 * G2m1 + alpha_2 * G1m1) + alpha_1 * e.g1 * e.pi1 * G2m1 + alpha_2 * e.g2 * e.pi2 * G1m1, G1m1 * G2m1, e.r_g12);
        double E = ei + 0.5 * rho * (u * u + v * v);
        double un = u * nx + v * ny;
        dv.pos(rho_1); dv.pos(rho_2); dv.mag(p + e.pi1); dv.mag(p + e.pi2); dv.mag(alpha_1);
        double a1_sq = dv(e.g1 * (p + e.pi1), rho_1);
        double a2_sq = dv(e.g2 * (p + e.pi2), rho_2);
        const double a_den = rho * (alpha_2 * rho_1 * a1_sq + alpha_1 * rho_2 * a2_sq);
        dv.den(a_den);
        double a_sq = dv(rho_1 * a1_sq * rho_2 * a2_sq, a_den);
        bad |= (a_sq < PRS_FLOOR);
        F[0] = alpha_1 * rho_1 * un;
        F[1] = alpha_2 * rho_2 * un;
        F[2] = rho * u * un + p * nx;
        F[3] = rho * v * un + p * ny;
        F[4] = (E + p) * un;
        F[5] = 0.0;
        return fabs(un) + sqrt(a_sq);
    }
    // kapila_5eqn.c:417-444
    template <class Dv>
    __device__ __forceinline__ static void ncp(const EosBase &e, Dv &dv, const double *V, const double *gx, const double *gy, double *B)
    {
        double alpha_1 = V[5];
        double alpha_2 = 1.0 - alpha_1;
        double rho_1 = V[0], rho_2 = V[1], u = V[2], v = V[3], p = V[4];
        double phi_x = gx[5], phi_y = gy[5];
        double u_x = gx[2], v_y = gy[3];
        dv.pos(rho_1); dv.pos(rho_2); dv.mag(p + e.pi1); dv.mag(p + e.pi2); dv.mag(alpha_1);
        double a_1_sq = dv(e.g1 * (p + e.pi1), rho_1);
        double a_2_sq = dv(e.g2 * (p + e.pi2), rho_2);
        const double k_den = alpha_1 * rho_2 * a_2_sq + alpha_2 * rho_1 * a_1_sq;
        dv.den(k_den);
        double K = dv(alpha_1 * alpha_2 * (rho_2 * a_2_sq - rho_1 * a_1_sq), k_den);
        B[0] = 0.0; B[1] = 0.0; B[2] = 0.0; B[3] = 0.0; B[4] = 0.0;
        B[5] = u * phi_x + v * phi_y - K * (u_x + v_y);
    }
    static constexpr bool ncp_nonzero(int c) { return c == 5; }
    static constexpr int order(int k) { constexpr int o[6] = {5, 2, 3, 4, 0, 1}; return o[k]; }
    // With rho_k in [2^-30, 2^16), p in [2^-20, 2^100), alpha_1 in [0, 1), 1 <= gamma <= 2^10 and
    // 0 <= pi <= 2^100: rho >= 2^-32 > RHO_FLOOR; rho_k a_k^2 = gamma_k (p + pi_k) >= 2^-20 and the
    // mixture's rho a^2 is at least the smaller of the two, so a^2 >= 2^-20 / 2^16 > PRS_FLOOR with
    // room for rounding; no product of pad() leaves [2^-400, 2^400]
    __device__ __forceinline__ static bool quick_eos(const EosBase &e)
    {
        return e.g1 >= 1.0 && e.g1 <= 1024.0 && e.g2 >= 1.0 && e.g2 <= 1024.0 && e.pi1 >= 0.0 && e.pi1 <= 0x1p100 &&
               e.pi2 >= 0.0 && e.pi2 <= 0x1p100;
    }
    template <int C>
    __device__ __forceinline__ static bool pad_quick(double v)
    {
        if constexpr (C <= 1) return exp_in<-30, 16>(v);
        else if constexpr (C == 4) return exp_in<-20, 100>(v);
        else if constexpr (C == 5) return frac_in(v);
        else return true;
    }
    // kapila_5eqn.c:450-479 (every test rejects: the one without a division first)
    template <class Dv>
    __device__ __forceinline__ static bool pad_dv(const EosBase &e, Dv &dv, const double *V)
    {
        double alpha_1 = V[5];
        if (alpha_1 < 0.0 || alpha_1 > 1.0) return false;
        double alpha_2 = 1.0 - alpha_1;
        double rho_1 = V[0], rho_2 = V[1];
        double rho = alpha_1 * rho_1 + alpha_2 * rho_2;
        double p = V[4];
        dv.pos(rho_1); dv.pos(rho_2); dv.mag(p + e.pi1); dv.mag(p + e.pi2); dv.mag(alpha_1);
        double a1_sq = dv(e.g1 * (p + e.pi1), rho_1);
        double a2_sq = dv(e.g2 * (p + e.pi2), rho_2);
        const double a_den = rho * (alpha_2 * rho_1 * a1_sq + alpha_1 * rho_2 * a2_sq);
        dv.den(a_den);
        double a_sq = dv(rho_1 * a1_sq * rho_2 * a2_sq, a_den);
        if (rho < RHO_FLOOR) return false;
        if (a_sq < PRS_FLOOR) return false;
        return true;
    }
    __device__ __forceinline__ static bool pad(const EosBase &e, const double *V)
    {
        IeeeDiv dv;
        return pad_dv(e, dv, V);
    }

    // ---- viscous fluxes (the VISCOUS build, hype.h:36) ----
    // kapila_5eqn.c:377-411: from primitive values V and gradients g[c][dim]
    // (only u, v: g[2], g[3] are read); returns the viscous eigenvalue
    template <int DIR>
    __device__ __forceinline__ static double visc_prim(const double *V, const double (*g)[2], double mu1, double mu2, double *F)
    {
        constexpr double nx = DIR == 0 ? 1.0 : 0.0, ny = DIR == 0 ? 0.0 : 1.0;
        const double r2_3 = 2. / 3., r4_3 = 4. / 3.;
        double phi = V[5];
        double mu = phi * mu1 + (1.0 - phi) * mu2;
        double u = V[2];
        double v = V[3];
        double u_x = g[2][0], u_y = g[2][1], v_x = g[3][0], v_y = g[3][1];
        double div_v = u_x + v_y;
        double tau_xx = mu * (2.0 * u_x - r2_3 * div_v);
        double tau_xy = mu * (u_y + v_x);
        double tau_yy = mu * (2.0 * v_y - r2_3 * div_v);
        F[0] = 0.0;
        F[1] = 0.0;
        F[2] = -nx * tau_xx - ny * tau_xy;
        F[3] = -nx * tau_xy - ny * tau_yy;
        F[4] = -nx * (u * tau_xx + v * tau_xy) - ny * (u * tau_xy + v * tau_yy);
        F[5] = 0.0;
        return r4_3 * mu / V[0];
    }
    // kapila_5eqn.c:119-158: from conserved values Q and their gradients (g[0..3] read)
    template <int DIR>
    __device__ __forceinline__ static double visc_cons(const double *Q, const double (*g)[2], double mu1, double mu2, double *F)
    {
        constexpr double nx = DIR == 0 ? 1.0 : 0.0, ny = DIR == 0 ? 0.0 : 1.0;
        const double r2_3 = 2. / 3., r4_3 = 4. / 3.;
        double phi = Q[5];
        double mu = phi * mu1 + (1.0 - phi) * mu2;
        double irho = 1.0 / (Q[0] + Q[1]);
        double u = irho * Q[2];
        double v = irho * Q[3];
        double rho_x = g[0][0] + g[1][0];
        double rho_y = g[0][1] + g[1][1];
        double u_x = irho * (g[2][0] - u * rho_x);
        double u_y = irho * (g[2][1] - u * rho_y);
        double v_x = irho * (g[3][0] - v * rho_x);
        double v_y = irho * (g[3][1] - v * rho_y);
        double div_v = u_x + v_y;
        double tau_xx = mu * (2.0 * u_x - r2_3 * div_v);
        double tau_xy = mu * (u_y + v_x);
        double tau_yy = mu * (2.0 * v_y - r2_3 * div_v);
        F[0] = 0.0;
        F[1] = 0.0;
        F[2] = -nx * tau_xx - ny * tau_xy;
        F[3] = -nx * tau_xy - ny * tau_yy;
        F[4] = -nx * (u * tau_xx + v * tau_xy) - ny * (u * tau_xy + v * tau_yy);
        F[5] = 0.0;
        return r4_3 * mu * irho;
    }

    // ---- conservative-variable path (RHSFunction, rhs_function.c) ----
    // kapila_5eqn.c:67-113
    template <int DIR>
    __device__ __forceinline__ static double flux_cons(const EosBase &e, const double *Q, double *F, bool &bad)
    {
        constexpr double nx = DIR == 0 ? 1.0 : 0.0, ny = DIR == 0 ? 0.0 : 1.0;
        double alpha_1 = Q[5];
        double alpha_2 = 1.0 - alpha_1;
        double rho_1 = Q[0] / alpha_1;
        double rho_2 = Q[1] / alpha_2;
        double rho = Q[0] + Q[1];
        double u = Q[2] / rho;
        double v = Q[3] / rho;
        double E = Q[4];
        double ei = E - 0.5 * rho * (u * u + v * v);
        double G1m1 = e.g1 - 1.0;
        double G2m1 = e.g2 - 1.0;
        double p = (ei * G1m1 * G2m1 - alpha_1 * e.g1 * e.pi1 * G2m1 - alpha_2 * e.g2 * e.pi2 * G1m1) / (alpha_1 * G2m1 + alpha_2 * G1m1);
        double un = u * nx + v * ny;
        double a1_sq = e.g1 * (p + e.pi1) / rho_1;
        double a2_sq = e.g2 * (p + e.pi2) / rho_2;
        double a_sq = (rho_1 * a1_sq * rho_2 * a2_sq) / (rho * (alpha_2 * rho_1 * a1_sq + alpha_1 * rho_2 * a2_sq));
        bad |= (a_sq < PRS_FLOOR);
        F[0] = alpha_1 * rho_1 * un;
        F[1] = alpha_2 * rho_2 * un;
        F[2] = rho * u * un + p * nx;
        F[3] = rho * v * un + p * ny;
        F[4] = (E + p) * un;
        F[5] = 0.0;
        return fabs(un) + sqrt(a_sq);
    }
    // kapila_5eqn.c:164-198
    __device__ __forceinline__ static void ncp_cons(const EosBase &e, const double *Q, const double *gx, const double *gy, double *B)
    {
        double alpha_1 = Q[5];
        double alpha_2 = 1.0 - alpha_1;
        double rho_1 = Q[0] / alpha_1;
        double rho_2 = Q[1] / alpha_2;
        double rho = Q[0] + Q[1];
        double irho = 1.0 / rho;
        double u = Q[2] / rho;
        double v = Q[3] / rho;
        double E = Q[4];
        double ei = E - 0.5 * rho * (u * u + v * v);
        double G1m1 = e.g1 - 1.0;
        double G2m1 = e.g2 - 1.0;
        double p = (ei * G1m1 * G2m1 - alpha_1 * e.g1 * e.pi1 * G2m1 - alpha_2 * e.g2 * e.pi2 * G1m1) / (alpha_1 * G2m1 + alpha_2 * G1m1);
        double a1_sq = e.g1 * (p + e.pi1) / rho_1;
        double a2_sq = e.g2 * (p + e.pi2) / rho_2;
        double K = alpha_1 * alpha_2 * (rho_2 * a2_sq - rho_1 * a1_sq) / (alpha_1 * rho_2 * a2_sq + alpha_2 * rho_1 * a1_sq);
        double alpha1_x = gx[5], alpha1_y = gy[5];
        double u_x = irho * irho * (gx[2] * rho - Q[2] * (gx[0] + gx[1]));
        double v_y = irho * irho * (gy[3] * rho - Q[3] * (gy[0] + gy[1]));
        B[0] = 0.0; B[1] = 0.0; B[2] = 0.0; B[3] = 0.0; B[4] = 0.0;
        B[5] = u * alpha1_x + v * alpha1_y - K * (u_x + v_y);
    }
    static constexpr bool ncp_cons_nonzero(int c) { return c == 5; }
    // a node value of alpha_1 that does not refuse the cell by itself: pad_cons's first test
    static constexpr int CONS_SCREEN = 5;
    __device__ __forceinline__ static bool cons_screen(double alpha_1) { return !(alpha_1 < 1.0 || alpha_1 > 1.0); }
    // kapila_5eqn.c:247-283; its alpha test (line 278) rejects every alpha_1 != 1
    __device__ __forceinline__ static bool pad_cons(const EosBase &e, const double *Q)
    {
        double alpha_1 = Q[5];
        if (alpha_1 < 1.0 || alpha_1 > 1.0) return false;   // every test rejects: the cheap one first
        double alpha_2 = 1.0 - alpha_1;
        double rho_1 = Q[0] / alpha_1;
        double rho_2 = Q[1] / alpha_2;
        double rho = Q[0] + Q[1];
        double u = Q[2] / rho;
        double v = Q[3] / rho;
        double E = Q[4];
        double ei = E - 0.5 * rho * (u * u + v * v);
        double G1m1 = e.g1 - 1.0;
        double G2m1 = e.g2 - 1.0;
        double p = (ei * G1m1 * G2m1 - alpha_1 * e.g1 * e.pi1 * G2m1 - alpha_2 * e.g2 * e.pi2 * G1m1) / (alpha_1 * G2m1 + alpha_2 * G1m1);
        double a1_sq = e.g1 * (p + e.pi1) / rho_1;
        double a2_sq = e.g2 * (p + e.pi2) / rho_2;
        double a_sq = (rho_1 * a1_sq * rho_2 * a2_sq) / (rho * (alpha_2 * rho_1 * a1_sq + alpha_1 * rho_2 * a2_sq));
        if (rho < RHO_FLOOR) return false;
        if (a_sq < PRS_FLOOR) return false;
        return true;
    }
};

// baer_nunziato.c: cons [a1 r1, a1 r1 u1, a1 r1 v1, a1 E1, a2 r2, a2 r2 u2, a2 r2 v2, a2 E2, a1]
//                  prim [r1, u1, v1, p1, r2, u2, v2, p2, a1]
template <> struct System<SYS_BN> {
    static constexpr int NV = 9;
    static constexpr int RX0 = 1, RX1 = 5, RY0 = 2, RY1 = 6;   // rhs_function_prim.c:115-117, 244-246
    // baer_nunziato.c:14-41
    __device__ __forceinline__ static void cons2prim(const EosBase &e, const double *Q, double *V)
    {
        IeeeDiv dv;
        cons2prim_dv(e, Q, V, dv);
    }
    template <class Dv>
    __device__ __forceinline__ static void cons2prim_dv(const EosBase &e, const double *Q, double *V, Dv &dv)
    {
        double phi_1 = Q[8];
        double phi_2 = 1.0 - Q[8];
        dv.frac(phi_1); dv.pos(Q[0]); dv.pos(Q[4]);
        dv.num(Q[1]); dv.num(Q[2]); dv.num(Q[3]); dv.num(Q[5]); dv.num(Q[6]); dv.num(Q[7]);
        const double y1 = dv.rcp(phi_1), y2 = dv.rcp(phi_2), z1 = dv.rcp(Q[0]), z2 = dv.rcp(Q[4]);
        double rho_1 = dv.quot(Q[0], phi_1, y1);
        double rho_2 = dv.quot(Q[4], phi_2, y2);
        double u_1 = dv.quot(Q[1], Q[0], z1), v_1 = dv.quot(Q[2], Q[0], z1);
        double u_2 = dv.quot(Q[5], Q[4], z2), v_2 = dv.quot(Q[6], Q[4], z2);
        double E_1 = dv.quot(Q[3], phi_1, y1);
        double E_2 = dv.quot(Q[7], phi_2, y2);
        double p_1 = (e.g1 - 1.0) * (E_1 - 0.5 * rho_1 * (u_1 * u_1 + v_1 * v_1)) - e.g1 * e.pi1;
        double p_2 = (e.g2 - 1.0) * (E_2 - 0.5 * rho_2 * (u_2 * u_2 + v_2 * v_2)) - e.g2 * e.pi2;
        V[0] = rho_1; V[1] = u_1; V[2] = v_1; V[3] = p_1;
        V[4] = rho_2; V[5] = u_2; V[6] = v_2; V[7] = p_2;
        V[8] = phi_1;
    }
    // baer_nunziato.c:47-60
    template <class Dv>
    __device__ __forceinline__ static void prim2cons(const EosBase &e, Dv &dv, const double *V, double *Q)
    {
        Q[0] = V[8] * V[0];
        Q[1] = Q[0] * V[1];
        Q[2] = Q[0] * V[2];
        Q[3] = Q[0] * (0.5 * (V[1] * V[1] + V[2] * V[2]) + dv(V[3] + e.g1 * e.pi1, V[0] * (e.g1 - 1.0)));
        Q[4] = (1.0 - V[8]) * V[4];
        Q[5] = Q[4] * V[5];
        Q[6] = Q[4] * V[6];
        Q[7] = Q[4] * (0.5 * (V[5] * V[5] + V[6] * V[6]) + dv(V[7] + e.g2 * e.pi2, V[4] * (e.g2 - 1.0)));
        Q[8] = V[8];
    }
    // baer_nunziato.c:256-321 (phase-2 flux pressure from V[8] unless fix_p2)
    template <int DIR, class Dv>
    __device__ __forceinline__ static double flux(const EosBase &e, Dv &dv, const double *V, double *F, bool &bad)
    {
        constexpr double nx = DIR == 0 ? 1.0 : 0.0, ny = DIR == 0 ? 0.0 : 1.0;
        double phi_1 = V[8];
        double phi_2 = 1.0 - V[8];
        double rho_1 = V[0], rho_2 = V[4];
        double u_1 = V[1], v_1 = V[2];
        double u_2 = V[5], v_2 = V[6];
        double p_1 = V[3];
        double p_2 = e.fix_p2 ? V[7] : V[8];
        dv.pos(rho_1); dv.pos(rho_2); dv.pos(p_1 + e.pi1); dv.pos(p_2 + e.pi2); dv.pos(V[7] + e.g2 * e.pi2);
        double E_1 = dv.by_const(p_1 + e.g1 * e.pi1, e.g1 - 1.0, e.r_g1) + 0.5 * rho_1 * (u_1 * u_1 + v_1 * v_1);
        double E_2 = dv.by_const(p_2 + e.g2 * e.pi2, e.g2 - 1.0, e.r_g2) + 0.5 * rho_2 * (u_2 * u_2 + v_2 * v_2);
        double un_1 = nx * u_1 + ny * v_1;
        double un_2 = nx * u_2 + ny * v_2;
        bad |= (rho_1 < RHO_FLOOR) | (rho_2 < RHO_FLOOR) | ((p_1 + e.pi1) < PRS_FLOOR) | ((p_2 + e.pi2) < PRS_FLOOR);
        F[0] = phi_1 * rho_1 * un_1;
        F[1] = phi_1 * (rho_1 * u_1 * un_1 + nx * p_1);
        F[2] = phi_1 * (rho_1 * v_1 * un_1 + ny * p_1);
        F[3] = phi_1 * un_1 * (E_1 + p_1);
        F[4] = phi_2 * rho_2 * un_2;
        F[5] = phi_2 * (rho_2 * u_2 * un_2 + nx * p_2);
        F[6] = phi_2 * (rho_2 * v_2 * un_2 + ny * p_2);
        F[7] = phi_2 * un_2 * (E_2 + p_2);
        F[8] = 0.0;
        double s_1 = fabs(un_1) + sqrt(dv(e.g1 * (p_1 + e.pi1), rho_1));
        double s_2 = fabs(un_2) + sqrt(dv(e.g2 * (p_2 + e.pi2), rho_2));
        return (s_1 < s_2) ? s_2 : s_1;
    }
    // baer_nunziato.c:327-344
    template <class Dv>
    __device__ __forceinline__ static void ncp(const EosBase &, Dv &, const double *V, const double *gx, const double *gy, double *B)
    {
        double u_I = V[1], v_I = V[2];
        double p_I = V[7];
        double phi_x = gx[8], phi_y = gy[8];
        B[0] = 0.0;
        B[1] = -p_I * phi_x;
        B[2] = -p_I * phi_y;
        B[3] = -p_I * (u_I * phi_x + v_I * phi_y);
        B[4] = 0.0;
        B[5] = p_I * phi_x;
        B[6] = p_I * phi_y;
        B[7] = p_I * (u_I * phi_x + v_I * phi_y);
        B[8] = u_I * phi_x + v_I * phi_y;
    }
    static constexpr bool ncp_nonzero(int c) { return c != 0 && c != 4; }
    static constexpr int order(int k) { constexpr int o[9] = {8, 1, 2, 7, 0, 3, 4, 5, 6}; return o[k]; }
    // rho_k >= 2^-30 > RHO_FLOOR, p_k >= 2^-20 and pi_k >= 0: p_k + pi_k > PRS_FLOOR, alpha_1 in [0, 1)
    __device__ __forceinline__ static bool quick_eos(const EosBase &e) { return e.pi1 >= 0.0 && e.pi2 >= 0.0; }
    template <int C>
    __device__ __forceinline__ static bool pad_quick(double v)
    {
        if constexpr (C == 0 || C == 4) return exp_in<-30, 1000>(v);
        else if constexpr (C == 3 || C == 7) return exp_in<-20, 1000>(v);
        else if constexpr (C == 8) return frac_in(v);
        else return true;
    }
    // baer_nunziato.c:350-385
    __device__ __forceinline__ static bool pad(const EosBase &e, const double *V)
    {
        bool ok = true;
        if (V[0] < RHO_FLOOR) ok = false;
        if (V[4] < RHO_FLOOR) ok = false;
        if ((V[3] + e.pi1) < PRS_FLOOR) ok = false;
        if ((V[7] + e.pi2) < PRS_FLOOR) ok = false;
        if (V[8] < 0.0 || V[8] > 1.0) ok = false;
        return ok;
    }

    // ---- conservative-variable path (RHSFunction, rhs_function.c) ----
    // baer_nunziato.c:66-131
    template <int DIR>
    __device__ __forceinline__ static double flux_cons(const EosBase &e, const double *Q, double *F, bool &bad)
    {
        constexpr double nx = DIR == 0 ? 1.0 : 0.0, ny = DIR == 0 ? 0.0 : 1.0;
        double phi_1 = Q[8];
        double phi_2 = 1.0 - Q[8];
        double rho_1 = Q[0] / phi_1;
        double rho_2 = Q[4] / phi_2;
        double u_1 = Q[1] / Q[0], v_1 = Q[2] / Q[0];
        double u_2 = Q[5] / Q[4], v_2 = Q[6] / Q[4];
        double E_1 = Q[3] / phi_1;
        double E_2 = Q[7] / phi_2;
        double p_1 = (e.g1 - 1.0) * (E_1 - 0.5 * rho_1 * (u_1 * u_1 + v_1 * v_1)) - e.g1 * e.pi1;
        double p_2 = (e.g2 - 1.0) * (E_2 - 0.5 * rho_2 * (u_2 * u_2 + v_2 * v_2)) - e.g2 * e.pi2;
        double un_1 = nx * u_1 + ny * v_1;
        double un_2 = nx * u_2 + ny * v_2;
        bad |= (rho_1 < RHO_FLOOR) | (rho_2 < RHO_FLOOR) | ((p_1 + e.pi1) < PRS_FLOOR) | ((p_2 + e.pi2) < PRS_FLOOR);
        F[0] = phi_1 * rho_1 * un_1;
        F[1] = phi_1 * (rho_1 * u_1 * un_1 + nx * p_1);
        F[2] = phi_1 * (rho_1 * v_1 * un_1 + ny * p_1);
        F[3] = phi_1 * un_1 * (E_1 + p_1);
        F[4] = phi_2 * rho_2 * un_2;
        F[5] = phi_2 * (rho_2 * u_2 * un_2 + nx * p_2);
        F[6] = phi_2 * (rho_2 * v_2 * un_2 + ny * p_2);
        F[7] = phi_2 * un_2 * (E_2 + p_2);
        F[8] = 0.0;
        double s_1 = fabs(un_1) + sqrt(e.g1 * (p_1 + e.pi1) / rho_1);
        double s_2 = fabs(un_2) + sqrt(e.g2 * (p_2 + e.pi2) / rho_2);
        return (s_1 < s_2) ? s_2 : s_1;
    }
    // baer_nunziato.c:137-165: u_I = u_1, p_I = p_2 from the phase-2 state
    __device__ __forceinline__ static void ncp_cons(const EosBase &e, const double *Q, const double *gx, const double *gy, double *B)
    {
        double phi_2 = 1.0 - Q[8];
        double rho_2 = Q[4] / phi_2;
        double u_1 = Q[1] / Q[0], v_1 = Q[2] / Q[0];
        double u_2 = Q[5] / Q[4], v_2 = Q[6] / Q[4];
        double E_2 = Q[7] / phi_2;
        double p_I = (e.g2 - 1.0) * (E_2 - 0.5 * rho_2 * (u_2 * u_2 + v_2 * v_2)) - e.g2 * e.pi2;
        double phi_x = gx[8], phi_y = gy[8];
        B[0] = 0.0;
        B[1] = -p_I * phi_x;
        B[2] = -p_I * phi_y;
        B[3] = -p_I * (u_1 * phi_x + v_1 * phi_y);
        B[4] = 0.0;
        B[5] = p_I * phi_x;
        B[6] = p_I * phi_y;
        B[7] = p_I * (u_1 * phi_x + v_1 * phi_y);
        B[8] = u_1 * phi_x + v_1 * phi_y;
    }
    static constexpr bool ncp_cons_nonzero(int c) { return c != 0 && c != 4; }
    static constexpr int CONS_SCREEN = -1;   // pad_cons has no test of one variable
    __device__ __forceinline__ static bool cons_screen(double) { return true; }
    // baer_nunziato.c:207-250
    __device__ __forceinline__ static bool pad_cons(const EosBase &e, const double *Q)
    {
        bool ok = true;
        double phi_1 = Q[8];
        double phi_2 = 1.0 - Q[8];
        double rho_1 = Q[0] / phi_1;
        double rho_2 = Q[4] / phi_2;
        double u_1 = Q[1] / Q[0], v_1 = Q[2] / Q[0];
        double u_2 = Q[5] / Q[4], v_2 = Q[6] / Q[4];
        double E_1 = Q[3] / phi_1;
        double E_2 = Q[7] / phi_2;
        double p_1 = (e.g1 - 1.0) * (E_1 - 0.5 * rho_1 * (u_1 * u_1 + v_1 * v_1)) - e.g1 * e.pi1;
        double p_2 = (e.g2 - 1.0) * (E_2 - 0.5 * rho_2 * (u_2 * u_2 + v_2 * v_2)) - e.g2 * e.pi2;
        if (rho_1 < RHO_FLOOR) ok = false;
        if (rho_2 < RHO_FLOOR) ok = false;
        if ((p_1 + e.pi1) < PRS_FLOOR) ok = false;
        if ((p_2 + e.pi2) < PRS_FLOOR) ok = false;
        if (phi_1 < 0.0 || phi_1 > 1.0) ok = false;
        return ok;
    }
};

// euler.c: cons [rho, rho u, rho v, E], prim [rho, u, v, p], ideal gas GAMMA_1
template <> struct System<SYS_EULER> {
    static constexpr int NV = 4;
    static constexpr int RX0 = 1, RX1 = -1, RY0 = 2, RY1 = -1;   // rhs_function_prim.c:101-102, 230-231
    // euler.c:14-23
    __device__ __forceinline__ static void cons2prim(const EosBase &e, const double *Q, double *V)
    {
        double irho = 1.0 / Q[0];
        V[0] = Q[0];
        V[1] = irho * Q[1];
        V[2] = irho * Q[2];
        V[3] = (e.g1 - 1.0) * (Q[3] - 0.5 * irho * (Q[1] * Q[1] + Q[2] * Q[2]));
    }
    // euler.c:29-38
    template <class Dv>
    __device__ __forceinline__ static void prim2cons(const EosBase &e, Dv &dv, const double *V, double *Q)
    {
        double ei = dv.by_const(V[3], e.g1 - 1.0, e.r_g1);
        double k = 0.5 * V[0] * (V[1] * V[1] + V[2] * V[2]);
        Q[0] = V[0];
        Q[1] = V[0] * V[1];
        Q[2] = V[0] * V[2];
        Q[3] = k + ei;
    }
    // euler.c:197-236
    template <int DIR, class Dv>
    __device__ __forceinline__ static double flux(const EosBase &e, Dv &dv, const double *V, double *F, bool &bad)
    {
        constexpr double nx = DIR == 0 ? 1.0 : 0.0, ny = DIR == 0 ? 0.0 : 1.0;
        double rho = V[0], u = V[1], v = V[2];
        double un = nx * u + ny * v;
        double rhoun = rho * un;
        double p = V[3];
        dv.pos(rho); dv.pos(p);
        double E = dv.by_const(p, e.g1 - 1.0, e.r_g1) + 0.5 * rho * (u * u + v * v);
        bad |= (rho < RHO_FLOOR) | (p < PRS_FLOOR);
        F[0] = rhoun;
        F[1] = rhoun * u + nx * p;
        F[2] = rhoun * v + ny * p;
        F[3] = un * (E + p);
        return fabs(un) + sqrt(dv(e.g1 * p, rho));
    }
    // euler.c:278-286
    template <class Dv>
    __device__ __forceinline__ static void ncp(const EosBase &, Dv &, const double *, const double *, const double *, double *B)
    {
        B[0] = 0.0; B[1] = 0.0; B[2] = 0.0; B[3] = 0.0;
    }
    static constexpr bool ncp_nonzero(int) { return false; }
    static constexpr int order(int k) { constexpr int o[4] = {0, 1, 2, 3}; return o[k]; }
    // rho >= 2^-30 > RHO_FLOOR, p >= 2^-30 > PRS_FLOOR
    __device__ __forceinline__ static bool quick_eos(const EosBase &) { return true; }
    template <int C>
    __device__ __forceinline__ static bool pad_quick(double v)
    {
        if constexpr (C == 0 || C == 3) return exp_in<-30, 1000>(v);
        else return true;
    }
    // euler.c:292-310
    __device__ __forceinline__ static bool pad(const EosBase &, const double *V)
    {
        bool ok = true;
        if (V[0] < RHO_FLOOR) ok = false;
        if (V[3] < PRS_FLOOR) ok = false;
        return ok;
    }

    // ---- conservative-variable path (RHSFunction, rhs_function.c) ----
    // euler.c:44-84
    template <int DIR>
    __device__ __forceinline__ static double flux_cons(const EosBase &e, const double *Q, double *F, bool &bad)
    {
        constexpr double nx = DIR == 0 ? 1.0 : 0.0, ny = DIR == 0 ? 0.0 : 1.0;
        double rho = Q[0];
        double irho = 1.0 / rho;
        double u = irho * Q[1];
        double v = irho * Q[2];
        double un = nx * u + ny * v;
        double rhoun = rho * un;
        double E = Q[3];
        double p = (e.g1 - 1.0) * (E - 0.5 * rho * (u * u + v * v));
        bad |= (rho < RHO_FLOOR) | (p < PRS_FLOOR);
        F[0] = rhoun;
        F[1] = rhoun * u + nx * p;
        F[2] = rhoun * v + ny * p;
        F[3] = un * (E + p);
        return fabs(un) + sqrt(e.g1 * p * irho);
    }
    __device__ __forceinline__ static void ncp_cons(const EosBase &, const double *, const double *, const double *, double *B)
    {
        B[0] = 0.0; B[1] = 0.0; B[2] = 0.0; B[3] = 0.0;
    }
    static constexpr bool ncp_cons_nonzero(int) { return false; }
    static constexpr int CONS_SCREEN = -1;
    __device__ __forceinline__ static bool cons_screen(double) { return true; }
    // euler.c:169-191
    __device__ __forceinline__ static bool pad_cons(const EosBase &e, const double *Q)
    {
        bool ok = true;
        double rho = Q[0];
        double irho = 1.0 / rho;
        double u = irho * Q[1];
        double v = irho * Q[2];
        double E = Q[3];
        double p = (e.g1 - 1.0) * (E - 0.5 * rho * (u * u + v * v));
        if (rho < RHO_FLOOR) ok = false;
        if (p < PRS_FLOOR) ok = false;
        return ok;
    }
};

// ---------------------------------------------------------------------------
// reconstruction (reconstruction.c)
// ---------------------------------------------------------------------------
struct Stencil {
    double c;
    double xm2, xm1, xp1, xp2;
    double ym2, ym1, yp1, yp2;
    double pp, pm, mp, mm;   // (i+1,j+1) (i+1,j-1) (i-1,j+1) (i-1,j-1)
};

// reconstruction.c:106-117
__device__ __forceinline__ double minmod(double a, double b)
{
    if (a * b < 0.0) return 0.0;
    return (fabs(a) < fabs(b)) ? a : b;
}
// reconstruction.c:123-127
__device__ __forceinline__ double pow4(double a) { double a2 = a * a; return a2 * a2; }

// reconstruction.c:157-178 for one direction
__device__ __forceinline__ void weno3_1d(double u_m2, double u_m1, double u_0, double u_p1, double u_p2, double &slope, double &curv)
{
    const double central_cell_wt = 100.0;
    double ux0 = -2.0 * u_m1 + 0.5 * u_m2 + 1.5 * u_0, uxx0 = 0.5 * (u_m2 - 2.0 * u_m1 + u_0);
    double ux1 = 0.5 * (u_p1 - u_m1),                  uxx1 = 0.5 * (u_m1 - 2.0 * u_0 + u_p1);
    double ux2 = -1.5 * u_0 + 2.0 * u_p1 - 0.5 * u_p2, uxx2 = 0.5 * (u_0 - 2.0 * u_p1 + u_p2);
    double IS0 = ux0 * ux0 + R13_3 * uxx0 * uxx0; double w0 = 1.0 / (pow4(IS0 + SMALL_NUM));
    double IS1 = ux1 * ux1 + R13_3 * uxx1 * uxx1; double w1 = central_cell_wt / (pow4(IS1 + SMALL_NUM));
    double IS2 = ux2 * ux2 + R13_3 * uxx2 * uxx2; double w2 = 1.0 / (pow4(IS2 + SMALL_NUM));
    double total = w0 + w1 + w2;
    w0 = w0 / total;
    w1 = w1 / total;
    w2 = w2 / total;
    slope = w0 * ux0 + w1 * ux1 + w2 * ux2;
    curv = w0 * uxx0 + w1 * uxx1 + w2 * uxx2;
}

// reconstruction.c:157-178 and :144-221 with the branch-free correctly rounded
// reciprocals and quotients of hype_div.cuh: the bits of weno3_1d / Recon<2>.  Every weight
// is gamma_k / d_k with d_k = (IS_k + 1e-12)^4 >= 1e-48 and is then divided by the weights'
// sum.  With every d_k below 2^400 all operands and quotients lie in div_rn's range; that is
// tested on the integer pipe, once per cell and variable.  Where the test fails (or for a NaN)
// `special` is set and the caller recomputes with Recon<2>.  The
// compiler's divisions each end in a branch, so a warp waits out one chain after the other;
// these interleave: Kapila 2048^2 right-hand side 1.76 -> 1.59 ms, BN 1024^2 0.896 -> 0.780,
// Euler 1531x897 0.380 -> 0.334.
struct CrCheck {
    unsigned hi = 0;
    __device__ __forceinline__ void divisor(double d) { hi = max(hi, (unsigned)__double2hiint(d)); }
    __device__ __forceinline__ bool special() const { return hi >= ((1023u + 400u) << 20); }
};

__device__ __forceinline__ void weno3_1d_cr(double u_m2, double u_m1, double u_0, double u_p1, double u_p2, double &slope,
                                            double &curv, CrCheck &ck)
{
    const double central_cell_wt = 100.0;
    // a product changes only its sign with its factor's: shared ones are formed once
    const double t_m1 = 2.0 * u_m1, t_0 = 2.0 * u_0, t_p1 = 2.0 * u_p1, s_0 = 1.5 * u_0;
    double ux0 = -t_m1 + 0.5 * u_m2 + s_0,  uxx0 = 0.5 * (u_m2 - t_m1 + u_0);
    double ux1 = 0.5 * (u_p1 - u_m1),       uxx1 = 0.5 * (u_m1 - t_0 + u_p1);
    double ux2 = -s_0 + t_p1 - 0.5 * u_p2,  uxx2 = 0.5 * (u_0 - t_p1 + u_p2);
    double IS0 = ux0 * ux0 + R13_3 * uxx0 * uxx0; const double d0 = pow4(IS0 + SMALL_NUM);
    double IS1 = ux1 * ux1 + R13_3 * uxx1 * uxx1; const double d1 = pow4(IS1 + SMALL_NUM);
    double IS2 = ux2 * ux2 + R13_3 * uxx2 * uxx2; const double d2 = pow4(IS2 + SMALL_NUM);
    ck.divisor(d0); ck.divisor(d1); ck.divisor(d2);
    double w0 = rcp_rn(d0);
    double w1 = div_rn(central_cell_wt, d1, rcp_rn(d1));
    double w2 = rcp_rn(d2);
    const double total = w0 + w1 + w2;
    const double y = rcp_rn(total);
    w0 = div_rn(w0, total, y);
    w1 = div_rn(w1, total, y);
    w2 = div_rn(w2, total, y);
    slope = w0 * ux0 + w1 * ux1 + w2 * ux2;
    curv = w0 * uxx0 + w1 * uxx1 + w2 * uxx2;
}
struct Recon2Cr {
    __device__ __forceinline__ static void run(const Stencil &s, double *c, bool &sp)
    {
        double u_0 = s.c;
        CrCheck ck;
        c[0] = u_0;
        weno3_1d_cr(s.xm2, s.xm1, u_0, s.xp1, s.xp2, c[1], c[3], ck);
        weno3_1d_cr(s.ym2, s.ym1, u_0, s.yp1, s.yp2, c[2], c[4], ck);
        double uxy0 =  s.pp - u_0 - c[1] - c[2] - c[3] - c[4];
        double uxy1 = -s.pm + u_0 + c[1] - c[2] + c[3] + c[4];
        double uxy2 = -s.mp + u_0 - c[1] + c[2] + c[3] + c[4];
        double uxy3 =  s.mm - u_0 + c[1] + c[2] - c[3] - c[4];
        double temp = 4.0 * (c[3] * c[3] + c[4] * c[4]);
        double IS0 = temp + uxy0 * uxy0; const double d0 = pow4(IS0 + SMALL_NUM);
        double IS1 = temp + uxy1 * uxy1; const double d1 = pow4(IS1 + SMALL_NUM);
        double IS2 = temp + uxy2 * uxy2; const double d2 = pow4(IS2 + SMALL_NUM);
        double IS3 = temp + uxy3 * uxy3; const double d3 = pow4(IS3 + SMALL_NUM);
        ck.divisor(d0); ck.divisor(d1); ck.divisor(d2); ck.divisor(d3);
        double w0 = rcp_rn(d0), w1 = rcp_rn(d1), w2 = rcp_rn(d2), w3 = rcp_rn(d3);
        const double total = w0 + w1 + w2 + w3;
        const double y = rcp_rn(total);
        w0 = div_rn(w0, total, y); w1 = div_rn(w1, total, y); w2 = div_rn(w2, total, y); w3 = div_rn(w3, total, y);
        c[5] = w0 * uxy0 + w1 * uxy1 + w2 * uxy2 + w3 * uxy3;
        sp = ck.special();
    }
};

template <int N> struct Recon;
template <> struct Recon<0> {
    __device__ __forceinline__ static void run(const Stencil &s, double *c) { c[0] = s.c; }
};
// reconstruction.c:129-142
template <> struct Recon<1> {
    __device__ __forceinline__ static void run(const Stencil &s, double *c)
    {
        c[0] = s.c;
        c[1] = minmod(s.xp1 - s.c, s.c - s.xm1);
        c[2] = minmod(s.yp1 - s.c, s.c - s.ym1);
    }
};
// reconstruction.c:144-221
template <> struct Recon<2> {
    __device__ __forceinline__ static void run(const Stencil &s, double *c)
    {
        double u_0 = s.c;
        c[0] = u_0;
        weno3_1d(s.xm2, s.xm1, u_0, s.xp1, s.xp2, c[1], c[3]);
        weno3_1d(s.ym2, s.ym1, u_0, s.yp1, s.yp2, c[2], c[4]);
        double uxy0 =  s.pp - u_0 - c[1] - c[2] - c[3] - c[4];
        double uxy1 = -s.pm + u_0 + c[1] - c[2] + c[3] + c[4];
        double uxy2 = -s.mp + u_0 - c[1] + c[2] + c[3] + c[4];
        double uxy3 =  s.mm - u_0 + c[1] + c[2] - c[3] - c[4];
        double temp = 4.0 * (c[3] * c[3] + c[4] * c[4]);
        double IS0 = temp + uxy0 * uxy0; double w0 = 1.0 / (pow4(IS0 + SMALL_NUM));
        double IS1 = temp + uxy1 * uxy1; double w1 = 1.0 / (pow4(IS1 + SMALL_NUM));
        double IS2 = temp + uxy2 * uxy2; double w2 = 1.0 / (pow4(IS2 + SMALL_NUM));
        double IS3 = temp + uxy3 * uxy3; double w3 = 1.0 / (pow4(IS3 + SMALL_NUM));
        double total = w0 + w1 + w2 + w3;
        w0 = w0 / total; w1 = w1 / total; w2 = w2 / total; w3 = w3 / total;
        c[5] = w0 * uxy0 + w1 * uxy1 + w2 * uxy2 + w3 * uxy3;
    }
};
// reconstruction.c:223-357.  CR: the weights' quotients by the branch-free forms, checked by
// `ck` (as Recon2Cr: every weight is gamma / d with d >= 1e-48 and then divided by the sum);
// Kapila 500^2 right-hand side 218 -> 196 us
struct Recon3 {
    template <bool CR>
    __device__ __forceinline__ static void weights(const Stencil &s, double *coeffs, CrCheck &ck)
    {
        auto over_d = [&](double g, double d) {
            if constexpr (CR) { ck.divisor(d); return div_rn(g, d, rcp_rn(d)); }
            else return g / d;
        };
        constexpr double gammaHi = 0.85, gammaLo = 0.85;
        double u_0 = s.c;
        double u_ip1 = s.xp1, u_jp1 = s.yp1, u_ip1jp1 = s.pp;
        double u_im1 = s.xm1, u_jm1 = s.ym1, u_ip1jm1 = s.pm;
        double u_ip2 = s.xp2, u_jp2 = s.yp2, u_im1jp1 = s.mp;
        double u_im2 = s.xm2, u_jm2 = s.ym2, u_im1jm1 = s.mm;
        double gamma_R4 = gammaHi;
        double gamma_R3[5];
        gamma_R3[0] = (1.0 - gammaHi) * gammaLo;
        for (int i = 1; i < 5; ++i) gamma_R3[i] = 0.25 * (1 - gammaHi) * (1 - gammaLo);
        double u_xR4 = R41_60 * (-u_im1 + u_ip1) + R11_120 * (u_im2 - u_ip2);
        double u_yR4 = R41_60 * (-u_jm1 + u_jp1) + R11_120 * (u_jm2 - u_jp2);
        double u_xxR4 = -u_0 + 0.5 * (u_im1 + u_ip1);
        double u_yyR4 = -u_0 + 0.5 * (u_jm1 + u_jp1);
        double u_xyR4 = 0.25 * (u_im1jm1 - u_im1jp1 - u_ip1jm1 + u_ip1jp1);
        double u_xxxR4 = R1_6 * (u_im1 - u_ip1) + R1_12 * (u_ip2 - u_im2);
        double u_yyyR4 = R1_6 * (u_jm1 - u_jp1) + R1_12 * (u_jp2 - u_jm2);
        double u_xxyR4 = 0.25 * (-u_im1jm1 + u_im1jp1 - u_ip1jm1 + u_ip1jp1) + 0.5 * (u_jm1 - u_jp1);
        double u_xyyR4 = 0.5 * (u_im1 - u_ip1) + 0.25 * (u_ip1jp1 - u_im1jm1 - u_im1jp1 + u_ip1jm1);
        double IS_R4 = (u_xR4 + 0.1 * u_xxxR4) * (u_xR4 + 0.1 * u_xxxR4) + R13_3 * (u_xxR4 * u_xxR4 + u_yyR4 * u_yyR4) +
                       (u_yR4 + 0.1 * u_yyyR4) * (u_yR4 + 0.1 * u_yyyR4) + 39.05 * (u_xxxR4 * u_xxxR4 + u_yyyR4 * u_yyyR4) +
                       R7_6 * u_xyR4 * u_xyR4 + 4.7 * (u_xxyR4 * u_xxyR4 + u_xyyR4 * u_xyyR4);
        double w_R4 = over_d(gamma_R4, pow4(IS_R4 + SMALL_NUM));
        double sum = w_R4;
        double u_xR3[5], u_yR3[5], u_xxR3[5], u_yyR3[5], u_xyR3[5], w_R3[5];
        u_xR3[0] = 0.5 * (-u_im1 + u_ip1);
        u_yR3[0] = 0.5 * (-u_jm1 + u_jp1);
        u_xxR3[0] = -u_0 + 0.5 * (u_im1 + u_ip1);
        u_yyR3[0] = -u_0 + 0.5 * (u_jm1 + u_jp1);
        u_xyR3[0] = 0.25 * (u_im1jm1 - u_im1jp1 - u_ip1jm1 + u_ip1jp1);
        u_xR3[1] = 1.5 * u_0 - 2.0 * u_im1 + 0.5 * u_im2;
        u_yR3[1] = 0.5 * (-u_jm1 + u_jp1);
        u_xxR3[1] = 0.5 * u_0 - u_im1 + 0.5 * u_im2;
        u_yyR3[1] = -u_0 + 0.5 * u_jm1 + 0.5 * u_jp1;
        u_xyR3[1] = 0.5 * (u_im1jm1 - u_im1jp1 - u_jm1 + u_jp1);
        u_xR3[2] = -1.5 * u_0 + 2.0 * u_ip1 - 0.5 * u_ip2;
        u_yR3[2] = 0.5 * (-u_jm1 + u_jp1);
        u_xxR3[2] = 0.5 * u_0 - u_ip1 + 0.5 * u_ip2;
        u_yyR3[2] = -u_0 + 0.5 * u_jm1 + 0.5 * u_jp1;
        u_xyR3[2] = 0.5 * (-u_ip1jm1 + u_ip1jp1 + u_jm1 - u_jp1);
        u_xR3[3] = 0.5 * (-u_im1 + u_ip1);
        u_yR3[3] = 1.5 * u_0 - 2.0 * u_jm1 + 0.5 * u_jm2;
        u_xxR3[3] = -u_0 + 0.5 * u_im1 + 0.5 * u_ip1;
        u_yyR3[3] = 0.5 * u_0 - u_jm1 + 0.5 * u_jm2;
        u_xyR3[3] = 0.5 * (-u_im1 + u_im1jm1 + u_ip1 - u_ip1jm1);
        u_xR3[4] = 0.5 * (-u_im1 + u_ip1);
        u_yR3[4] = -1.5 * u_0 + 2.0 * u_jp1 - 0.5 * u_jp2;
        u_xxR3[4] = -u_0 + 0.5 * u_im1 + 0.5 * u_ip1;
        u_yyR3[4] = 0.5 * u_0 - u_jp1 + 0.5 * u_jp2;
        u_xyR3[4] = 0.5 * (u_im1 - u_im1jp1 - u_ip1 + u_ip1jp1);
#pragma unroll
        for (int i = 0; i < 5; ++i) {
            double IS = u_xR3[i] * u_xR3[i] + u_yR3[i] * u_yR3[i] + R13_3 * (u_xxR3[i] * u_xxR3[i] + u_yyR3[i] * u_yyR3[i]) + R7_6 * u_xyR3[i] * u_xyR3[i];
            w_R3[i] = over_d(gamma_R3[i], pow4(IS + SMALL_NUM));
            sum += w_R3[i];
        }
        double wt_ratio;
        if constexpr (CR) {
            const double y = rcp_rn(sum);
            w_R4 = div_rn(w_R4, sum, y);
#pragma unroll
            for (int i = 0; i < 5; ++i) w_R3[i] = div_rn(w_R3[i], sum, y);
            constexpr double r_gamma = 1.0 / gammaHi;   // correctly rounded
            wt_ratio = div_rn(w_R4, gamma_R4, r_gamma);
        } else {
            w_R4 = w_R4 / sum;
#pragma unroll
            for (int i = 0; i < 5; ++i) w_R3[i] = w_R3[i] / sum;
            wt_ratio = w_R4 / gamma_R4;
        }
        coeffs[0] = u_0;
#define HYPE_W4(R4, R3) (wt_ratio * (R4 - gamma_R3[0] * R3[0] - gamma_R3[1] * R3[1] - gamma_R3[2] * R3[2] - gamma_R3[3] * R3[3] - gamma_R3[4] * R3[4]) \
                         + w_R3[0] * R3[0] + w_R3[1] * R3[1] + w_R3[2] * R3[2] + w_R3[3] * R3[3] + w_R3[4] * R3[4])
        coeffs[1] = HYPE_W4(u_xR4, u_xR3);
        coeffs[2] = HYPE_W4(u_yR4, u_yR3);
        coeffs[3] = HYPE_W4(u_xxR4, u_xxR3);
        coeffs[4] = HYPE_W4(u_yyR4, u_yyR3);
        coeffs[5] = HYPE_W4(u_xyR4, u_xyR3);
#undef HYPE_W4
        coeffs[6] = wt_ratio * u_xxxR4;
        coeffs[7] = wt_ratio * u_yyyR4;
        coeffs[8] = wt_ratio * u_xxyR4;
        coeffs[9] = wt_ratio * u_xyyR4;
    }
};
template <> struct Recon<3> {
    __device__ __forceinline__ static void run(const Stencil &s, double *c)
    {
        CrCheck ck;
        Recon3::weights<false>(s, c, ck);
    }
};
struct Recon3Cr {
    __device__ __forceinline__ static void run(const Stencil &s, double *c, bool &sp)
    {
        CrCheck ck;
        Recon3::weights<true>(s, c, ck);
        sp = ck.special();
    }
};
template <int N> using ReconCr = std::conditional_t<N == 2, Recon2Cr, Recon3Cr>;

// The unlimited central coefficients (u_coeffs) Reconstruct returns beside
// the WENO ones (reconstruction.c:139-141, 172-174, 195-196, 217, 258-267);
// the VISCOUS build takes face gradients from them.  N = 0: the reference
// leaves them unset, so the viscous path starts at N = 1.
template <int N> struct UCoef;
template <> struct UCoef<1> {
    __device__ __forceinline__ static void run(const Stencil &s, double *uc)
    {
        uc[0] = s.c;
        uc[1] = 0.5 * (s.xp1 - s.xm1);
        uc[2] = 0.5 * (s.yp1 - s.ym1);
    }
};
template <> struct UCoef<2> {
    __device__ __forceinline__ static void run(const Stencil &s, double *uc)
    {
        const double u_0 = s.c;
        uc[0] = u_0;
        uc[1] = 0.5 * (s.xp1 - s.xm1);
        uc[3] = 0.5 * (s.xm1 - 2.0 * u_0 + s.xp1);
        uc[2] = 0.5 * (s.yp1 - s.ym1);
        uc[4] = 0.5 * (s.ym1 - 2.0 * u_0 + s.yp1);
        uc[5] = 0.25 * (s.pp - s.pm - s.mp + s.mm);
    }
};
template <> struct UCoef<3> {
    __device__ __forceinline__ static void run(const Stencil &s, double *uc)
    {
        const double u_0 = s.c;
        const double u_ip1 = s.xp1, u_jp1 = s.yp1, u_ip1jp1 = s.pp, u_im1 = s.xm1, u_jm1 = s.ym1, u_ip1jm1 = s.pm;
        const double u_ip2 = s.xp2, u_jp2 = s.yp2, u_im1jp1 = s.mp, u_im2 = s.xm2, u_jm2 = s.ym2, u_im1jm1 = s.mm;
        uc[0] = u_0;
        uc[1] = R41_60 * (-u_im1 + u_ip1) + R11_120 * (u_im2 - u_ip2);
        uc[2] = R41_60 * (-u_jm1 + u_jp1) + R11_120 * (u_jm2 - u_jp2);
        uc[3] = -u_0 + 0.5 * (u_im1 + u_ip1);
        uc[4] = -u_0 + 0.5 * (u_jm1 + u_jp1);
        uc[5] = 0.25 * (u_im1jm1 - u_im1jp1 - u_ip1jm1 + u_ip1jp1);
        uc[6] = R1_6 * (u_im1 - u_ip1) + R1_12 * (u_ip2 - u_im2);
        uc[7] = R1_6 * (u_jm1 - u_jp1) + R1_12 * (u_jp2 - u_jm2);
        uc[8] = 0.25 * (-u_im1jm1 + u_im1jp1 - u_ip1jm1 + u_ip1jp1) + 0.5 * (u_jm1 - u_jp1);
        uc[9] = 0.5 * (u_im1 - u_ip1) + 0.25 * (u_ip1jp1 - u_im1jm1 - u_im1jp1 + u_ip1jm1);
    }
};

}  // namespace hype
