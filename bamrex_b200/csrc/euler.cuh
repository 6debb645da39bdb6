// Device-side Euler physics of the explicit path: primitive conversion,
// physical flux, slope limiters, MUSCL-Hancock cell stage, and the HLLC /
// FORCE / Lax-Friedrichs face stages, templated on the arithmetic type T
// (double: the drop-in path; float: the FP32-storage variant).  Each
// function follows the reference routine cited beside it in operation
// order, except that a reciprocal of the density (or of epsilon) is reused
// where the reference divides several times by the same value, and that the
// fast path evaluates the gamma powers of the Toro wave-speed estimate as a
// refined integer root.  In FP64 both change results by a few units in the
// last place (parity bound: 1e-12 relative L-infinity per step).
#pragma once

#include <cmath>

#include "common.cuh"

namespace bamrex {

enum { LIM_MINBEE = 0, LIM_VAN_LEER = 1, LIM_VAN_ALBADA = 2, LIM_SUPERBEE = 3 };
enum { M_MUSCL = 0, M_HLLC = 1, M_SLIC = 4, M_FORCE = 5, M_LF = 6 };

// Minimum density / pressure of the wave-speed estimate (HLLC.H:255-260).
constexpr double kMinRho = 1e-14;
constexpr double kMinP = 1e-14;

// The run constants in the arithmetic type of a kernel.
template <typename T>
struct K {
    T gamma, eps, inv_eps, gm1, half_gm1, z, neg_z, inv_z, gp1_2g, gamma_inv_eps, half_eps;
    T neg_gm1_heps, one_m_gp1_2g;  // -(gamma - 1) eps / 2 and 1 - (gamma + 1) / (2 gamma): the fast path
    double root_dneg_l2, root_dpos_l2, root_ik, root_c2;
    int root_k, limiter, uniform_var, need_prim;
    int lim_var[kMaxComp], lim_prim[kMaxComp];

    __device__ __forceinline__ explicit K(const Consts& c)
        : gamma((T)c.gamma), eps((T)c.eps), inv_eps((T)c.inv_eps), gm1((T)c.gm1), half_gm1((T)c.half_gm1),
          z((T)c.z), neg_z((T)c.neg_z), inv_z((T)c.inv_z), gp1_2g((T)c.gp1_2g), gamma_inv_eps((T)c.gamma_inv_eps),
          half_eps((T)c.half_eps), neg_gm1_heps((T)c.neg_gm1_heps), one_m_gp1_2g((T)c.one_m_gp1_2g),
          root_dneg_l2(c.root_dneg_l2), root_dpos_l2(c.root_dpos_l2), root_ik(c.root_ik), root_c2(c.root_c2), root_k(c.root_k),
          limiter(c.limiter), uniform_var(c.uniform_var), need_prim(c.need_prim)
    {
#pragma unroll
        for (int n = 0; n < kMaxComp; ++n) {
            lim_var[n] = c.lim_var[n];
            lim_prim[n] = c.lim_prim[n];
        }
    }
};

// a[idx] for a runtime idx without local-memory indexing.
template <typename T, int N>
__device__ __forceinline__ T sel(const T (&a)[N], int idx)
{
    T r = a[0];
#pragma unroll
    for (int m = 1; m < N; ++m) r = (idx == m) ? a[m] : r;
    return r;
}

template <int D, int DIR>
struct Prim;

// primv_from_consv (Source/System/Euler/Euler.H:167-198); inv_rho = 1/rho.
// FP32 spells out its multiply-adds (here and in phys_flux), as the compiler
// contracts them where nothing around competes for the products.
template <typename T, int D>
__device__ __forceinline__ void to_prim(const T (&U)[D + 2], const K<T>& k, T (&q)[D + 2], T& inv_rho)
{
    inv_rho = T(1) / U[0];
    q[0] = U[0];
#pragma unroll
    for (int d = 0; d < D; ++d) q[1 + d] = U[1 + d] * inv_rho;
    T usq;
    if constexpr (sizeof(T) == 4 && D > 1) {
        usq = fmaf(q[1], q[1], __fmul_rn(q[2], q[2]));
        if constexpr (D > 2) usq = fmaf(q[3], q[3], usq);
    } else {
        usq = q[1] * q[1];
#pragma unroll
        for (int d = 1; d < D; ++d) usq = usq + q[1 + d] * q[1 + d];
    }
    q[1 + D] = k.gm1 * (U[1 + D] - k.half_eps * U[0] * usq);
}

// euler_flux<dir> / compute_flux_function<dir> (Euler.H:211-244, Euler.cpp:10-44).
template <typename T, int D, int DIR>
__device__ __forceinline__ void phys_flux(const T (&U)[D + 2], const T (&q)[D + 2], const K<T>& k, T (&F)[D + 2])
{
    const T mn = U[1 + DIR];
    F[0] = mn;
#pragma unroll
    for (int d = 0; d < D; ++d) F[1 + d] = mn * q[1 + d];
    if constexpr (sizeof(T) == 4) F[1 + DIR] = fmaf(mn, q[1 + DIR], __fmul_rn(q[1 + D], k.inv_eps));
    else F[1 + DIR] += q[1 + D] * k.inv_eps;
    F[1 + D] = (U[1 + D] + q[1 + D]) * q[1 + DIR];
}

template <typename T, int D, int DIR>
__device__ __forceinline__ void phys_flux(const T (&U)[D + 2], const K<T>& k, T (&F)[D + 2])
{
    if constexpr (sizeof(T) == 8) {
        const Prim<D, DIR> q(U, k);
        F[0] = U[1 + DIR];
#pragma unroll
        for (int d = 0; d < D; ++d) F[1 + d] = d == DIR ? fma(q.p, k.inv_eps, q.mnu) : __dmul_rn(U[1 + DIR], q.u[d]);
        F[1 + D] = __dmul_rn(U[1 + D] + q.p, q.u[DIR]);
    } else {
        T q[D + 2], ir;
        to_prim<T, D>(U, k, q, ir);
        phys_flux<T, D, DIR>(U, q, k, F);
    }
}

// slope_limit<L> (Source/Fluxes/Limiters.H:29-73).
template <typename T>
__device__ __forceinline__ T slope_limit(int lim, T r)
{
    if (r <= T(0)) return T(0);
    switch (lim) {
    case LIM_MINBEE: return r > T(1) ? fmin(T(2) / (T(1) + r), T(1)) : r;
    case LIM_VAN_LEER: {
        const T ip = T(1) / (T(1) + r);
        return fmin(T(2) * r * ip, T(2) * ip);
    }
    case LIM_VAN_ALBADA: return fmin(r * (T(1) + r) / (T(1) + r * r), T(2) / (T(1) + r));
    default: return (r <= T(0.5)) ? T(2) * r : ((r <= T(1)) ? T(1) : fmin(r, fmin(T(2) / (T(1) + r), T(2))));
    }
}

// The limiter value from the limiting-variable differences
// (Source/Fluxes/Flux_Helpers.cpp:103-111).
template <typename T>
__device__ __forceinline__ T limiter_value(int lim, T numerator, T denom)
{
    if (numerator == T(0) && denom == T(0)) return slope_limit<T>(lim, T(1));
    if (denom == T(0)) return T(0);
    return slope_limit<T>(lim, numerator / denom);
}

// ---- cell stage: reconstruct_and_half_time_step<limiter,dir> --------------
// (general path of FP32 storage; FP64: muscl_cell_gen, hllc_face_f64<GEN>)
// (Source/Fluxes/Flux_Helpers.cpp:92-148) for one cell from its two
// neighbours along the sweep: returns the half-stepped L/R states.
template <typename T, int D, int DIR>
__device__ __forceinline__ void muscl_cell(const T (&Um)[D + 2], const T (&U0)[D + 2], const T (&Up)[D + 2],
                                           const K<T>& k, T hdtdx, T (&UL)[D + 2], T (&UR)[D + 2])
{
    constexpr int NC = D + 2;
    T hphi[NC];
    if (k.uniform_var >= 0) {
        const int v = k.uniform_var;
        const T vL = sel(Um, v), vC = sel(U0, v), vR = sel(Up, v);
        const T lim = limiter_value<T>(k.limiter, vC - vL, vR - vC);
#pragma unroll
        for (int n = 0; n < NC; ++n) hphi[n] = T(0.5) * lim;
    } else {
        T Qm[NC], Q0[NC], Qp[NC], ir;
        if (k.need_prim) {
            to_prim<T, D>(Um, k, Qm, ir);
            to_prim<T, D>(U0, k, Q0, ir);
            to_prim<T, D>(Up, k, Qp, ir);
        } else {
#pragma unroll
            for (int n = 0; n < NC; ++n) Qm[n] = Q0[n] = Qp[n] = T(0);
        }
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            const int v = k.lim_var[n];
            const bool pr = k.lim_prim[n] != 0;
            const T vL = pr ? sel(Qm, v) : sel(Um, v);
            const T vC = pr ? sel(Q0, v) : sel(U0, v);
            const T vR = pr ? sel(Qp, v) : sel(Up, v);
            hphi[n] = T(0.5) * limiter_value<T>(k.limiter, vC - vL, vR - vC);
        }
    }
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const T delta = T(0.5) * (U0[n] - Um[n]) + T(0.5) * (Up[n] - U0[n]);
        UL[n] = U0[n] - hphi[n] * delta;
        UR[n] = U0[n] + hphi[n] * delta;
    }
    T FL[NC], FR[NC];
    phys_flux<T, D, DIR>(UL, k, FL);
    phys_flux<T, D, DIR>(UR, k, FR);
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const T dF = hdtdx * (FR[n] - FL[n]);
        UL[n] -= dF;
        UR[n] -= dF;
    }
}

// ---- face stage: HLLC (Source/Fluxes/HLLC.cpp:90-172 with
// estimate_wave_speed_HLLC_Toro, HLLC.H:214-309, and
// HLLC_interm_state_replace, HLLC.H:311-337).  L is the state left of the
// face, R the state right of it.
template <typename T, int D, int DIR>
__device__ __forceinline__ void hllc_face(const T (&L)[D + 2], const T (&R)[D + 2], const K<T>& k, T (&F)[D + 2])
{
    constexpr int NC = D + 2;
    T qL[NC], qR[NC], irL, irR;
    to_prim<T, D>(L, k, qL, irL);
    to_prim<T, D>(R, k, qR, irR);
    const T rhoL = fmax(qL[0], T(kMinRho)), rhoR = fmax(qR[0], T(kMinRho));
    const T pL = fmax(qL[1 + D], T(kMinP)), pR = fmax(qR[1 + D], T(kMinP));
    const T uL = qL[1 + DIR], uR = qR[1 + DIR];
    const T icL = (qL[0] >= T(kMinRho)) ? irL : T(1.0 / kMinRho);
    const T icR = (qR[0] >= T(kMinRho)) ? irR : T(1.0 / kMinRho);
    const T cL = sqrt(k.gamma_inv_eps * pL * icL);
    const T cR = sqrt(k.gamma_inv_eps * pR * icR);
    const T base = (cL + cR - k.half_gm1 * (uR - uL)) / (cL * pow(pL, k.neg_z) + cR * pow(pR, k.neg_z));
    const T p_rr = pow(base, k.inv_z);
    const T qwL = (p_rr > pL) ? sqrt(T(1) + k.gp1_2g * (p_rr / pL - T(1))) : T(1);
    const T qwR = (p_rr > pR) ? sqrt(T(1) + k.gp1_2g * (p_rr / pR - T(1))) : T(1);
    const T SL = uL - cL * qwL;
    const T SR = uR + cR * qwR;
    const T dL = SL - uL, dR = SR - uR;
    const T denom = rhoL * dL - rhoR * dR;
    const T Ss = (denom != T(0)) ? ((pR - pL) * k.inv_eps + rhoL * uL * dL - rhoR * uR * dR) / denom : T(0);

    // Branches of HLLC.cpp:101-167: the left states serve when S_L >= 0 or
    // S* >= 0; the star correction applies unless the face is supersonic.
    const bool useL = (SL >= T(0)) || (Ss >= T(0));
    const bool star = useL ? (SL < T(0)) : (SR >= T(0));
    T UK[NC], qK[NC];
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        UK[n] = useL ? L[n] : R[n];
        qK[n] = useL ? qL[n] : qR[n];
    }
    const T irK = useL ? irL : irR;
    const T SK = useL ? SL : SR;
    phys_flux<T, D, DIR>(UK, qK, k, F);
    if (star) {
        const T rhoK = qK[0], uK = qK[1 + DIR], pK = qK[1 + D];
        const T dK = SK - uK;
        const T scale = rhoK * dK / (SK - Ss);
        const T eterm = UK[1 + D] * irK + (Ss - uK) * (Ss * k.eps + pK / (rhoK * dK));
        F[0] = F[0] + SK * (scale - UK[0]);
#pragma unroll
        for (int d = 0; d < D; ++d) {
            const T s = (d == DIR) ? Ss : qK[1 + d];
            F[1 + d] = F[1 + d] + SK * (s * scale - UK[1 + d]);
        }
        F[1 + D] = F[1 + D] + SK * (eterm * scale - UK[1 + D]);
    }
}

// FORCE and Lax-Friedrichs take the products of two neighbouring cells' fluxes
// into sums.  Every product and sum is spelled out, so that a face has the same
// bits in whichever kernel, and whichever position of a lane, it is formed (a
// level in boxes steps like one box); left to the compiler, the product that a
// sum is contracted with depends on how often each is used around it.
//
// a d + s / 2
__device__ __forceinline__ double centred_sum(double a, double d, double s) { return fma(a, d, 0.5 * s); }
__device__ __forceinline__ float centred_sum(float a, float d, float s) { return fmaf(a, d, 0.5f * s); }

// The sum and the difference of two states' fluxes.  FP32: each flux but the
// mass and the normal momentum is a product, and the right one (LEFT: the
// left one) enters unrounded, which are the bits FORCE and Lax-Friedrichs
// have always had.
template <int D, int DIR, bool LEFT>
__device__ __forceinline__ void flux_pair(const double (&L)[D + 2], const double (&R)[D + 2], const K<double>& k,
                                          double (&sum)[D + 2], double (&dif)[D + 2])
{
    double fL[D + 2], fR[D + 2];
    phys_flux<double, D, DIR>(L, k, fL);
    phys_flux<double, D, DIR>(R, k, fR);
#pragma unroll
    for (int n = 0; n < D + 2; ++n) {
        sum[n] = fL[n] + fR[n];
        dif[n] = fL[n] - fR[n];
    }
}
template <int D, int DIR, bool LEFT>
__device__ __forceinline__ void flux_pair(const float (&L)[D + 2], const float (&R)[D + 2], const K<float>& k,
                                          float (&sum)[D + 2], float (&dif)[D + 2])
{
    constexpr int E = D + 1;
    float qL[D + 2], qR[D + 2], ir;
    to_prim<float, D>(L, k, qL, ir);
    to_prim<float, D>(R, k, qR, ir);
    sum[0] = L[1 + DIR] + R[1 + DIR];
    dif[0] = L[1 + DIR] - R[1 + DIR];
#pragma unroll
    for (int n = 1; n < D + 2; ++n) {
        // the flux as x y
        const float xL = n == E ? L[E] + qL[E] : L[1 + DIR], yL = n == E ? qL[1 + DIR] : qL[n];
        const float xR = n == E ? R[E] + qR[E] : R[1 + DIR], yR = n == E ? qR[1 + DIR] : qR[n];
        if (n == 1 + DIR) {
            const float a = fmaf(xL, yL, __fmul_rn(qL[E], k.inv_eps)), b = fmaf(xR, yR, __fmul_rn(qR[E], k.inv_eps));
            sum[n] = a + b;
            dif[n] = a - b;
        } else if (LEFT) {
            sum[n] = fmaf(xL, yL, __fmul_rn(xR, yR));
            dif[n] = fmaf(xL, yL, -__fmul_rn(xR, yR));
        } else {
            sum[n] = fmaf(xR, yR, __fmul_rn(xL, yL));
            dif[n] = fmaf(-xR, yR, __fmul_rn(xL, yL));
        }
    }
}

// ---- face stage: FORCE (compute_force_flux_LR, Source/Fluxes/Force.cpp:22-108)
template <typename T, int D, int DIR>
__device__ __forceinline__ void force_face(const T (&L)[D + 2], const T (&R)[D + 2], const K<T>& k, T half_dx_dt,
                                           T dt_2dx, T (&F)[D + 2])
{
    constexpr int NC = D + 2;
    T sum[NC], dif[NC], H[NC], fH[NC];
    flux_pair<D, DIR, false>(L, R, k, sum, dif);
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        F[n] = T(0.5) * centred_sum(half_dx_dt, L[n] - R[n], sum[n]);
        if constexpr (sizeof(T) == 8) H[n] = centred_sum(dt_2dx, dif[n], L[n] + R[n]);
        else H[n] = fmaf(0.5f, L[n] + R[n], __fmul_rn(dt_2dx, dif[n]));
    }
    phys_flux<T, D, DIR>(H, k, fH);
#pragma unroll
    for (int n = 0; n < NC; ++n) F[n] += T(0.5) * fH[n];
}

// ---- face stage: Lax-Friedrichs (compute_LF_flux, Source/Fluxes/Force.cpp:110-151)
template <typename T, int D, int DIR>
__device__ __forceinline__ void lf_face(const T (&L)[D + 2], const T (&R)[D + 2], const K<T>& k, T half_dx_dt,
                                        T (&F)[D + 2])
{
    constexpr int NC = D + 2;
    T sum[NC], dif[NC];
    flux_pair<D, DIR, true>(L, R, k, sum, dif);
#pragma unroll
    for (int n = 0; n < NC; ++n) F[n] = centred_sum(half_dx_dt, L[n] - R[n], sum[n]);
}

// |u| + c of a conserved state (max_wave_speed body, Euler.cpp:53-68).
template <typename T, int D>
__device__ __forceinline__ T wave_speed(const T (&U)[D + 2], const K<T>& k)
{
    T q[D + 2], ir;
    to_prim<T, D>(U, k, q, ir);
    T vsq = q[1] * q[1];
#pragma unroll
    for (int d = 1; d < D; ++d) vsq = vsq + q[1 + d] * q[1 + d];
    return sqrt(k.gamma_inv_eps * q[1 + D] * ir) + sqrt(vsq);
}

// ======================================================================
// Fast path: MUSCL-Hancock + HLLC with a compile-time limiter, every
// component limited on the energy (the reference default,
// FluidSystem.cpp:65-69), and gamma with 1/z = 7 (gamma = 1.4).  Same
// arithmetic as above but branch-free (selects instead of branches), with
// refined reciprocals in FP64 and the hardware approximations in FP32, so
// each cell and face is one basic block the scheduler can interleave.
// ======================================================================

// 1/x.  FP64: the hardware approximation r (PTX rcp.approx.ftz.f64; its
// relative error measured below 2^-19.9 on the B200 over 2^30 arguments)
// refined by one third-order step of the series 1/x = r / (1 - e) with
// e = 1 - x r: r (1 + e + e^2), three fused multiply-adds; within 1 ulp of
// the correctly rounded quotient for normal, finite x (the same probe), as
// two Newton steps are, for one multiply-add less.  FP32: the hardware
// approximation.
__device__ __forceinline__ double rcp_fast(double x)
{
    double r;
    asm("rcp.approx.ftz.f64 %0, %1;" : "=d"(r) : "d"(x));
    const double e = fma(-x, r, 1.0);
    return fma(r, fma(e, e, e), r);
}
__device__ __forceinline__ float rcp_fast(float x)
{
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// FP32 special-function approximations (PTX .approx.ftz.f32, a few ulp):
// the FP32-storage variant reports its error against the FP64 oracle
// instead of holding a bit-level bar.
__device__ __forceinline__ float sqrt_fast(float x)
{
    float r;
    asm("sqrt.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// sqrt(x) for a positive, normal, finite x without the special-case branch of
// sqrt(): the coupled iteration for g ~ sqrt(x), h ~ 1 / (2 sqrt(x)) seeded
// by the hardware reciprocal square root (PTX rsqrt.approx.ftz.f64, relative
// error below 2^-19.9): one step g += g r with r = 1/2 - g h (relative error
// ~1.5 e^2, e the seed's), then the correction g += h (x - g^2) with the
// seed's h, whose own error only scales the already tiny correction
// (P. Markstein, IA-64 and Elementary Functions, 2000).  The seed is halved
// in its exponent field (an integer subtraction, off the FP64 pipe).  Zero,
// infinity and subnormal x give NaN.
__device__ __forceinline__ double sqrt_pos(double x)
{
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(x));
    const double g = x * y;
    const double h = __hiloint2double(__double2hiint(y) - 0x00100000, __double2loint(y));
    const double r = fma(-g, h, 0.5);
    const double g1 = fma(g, r, g);
    const double d = fma(-g1, g1, x);
    return fma(d, h, g1);
}

__device__ __forceinline__ float ex2_fast(float x)
{
    float r;
    asm("ex2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}
__device__ __forceinline__ float lg2_fast(float x)
{
    float r;
    asm("lg2.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// log2(x) of a positive normal double in single precision from its exponent
// field and the first 20 mantissa bits (absolute error below 2^-19 for the
// mantissa part): integer operations and one lg2, no conversion.
__device__ __forceinline__ float log2_hi(double x)
{
    const int hi = __double2hiint(x);
    const float ex = __int_as_float(0x4b400000 + ((hi >> 20) & 0x7ff)) - (12582912.0f + 1023.0f);
    return ex + lg2_fast(__int_as_float(0x3f800000 | ((hi & 0x000fffff) << 3)));
}

// w^(-1/7) and 1/w for a positive normal w.  FP64: seed y0 = 2^(-log2(w)/7)
// in single precision (relative error below 2^-20; its bits are moved into a
// double by integer operations), then one step of the series of
// (1 - e)^(-1/7), e = 1 - w y0^7 (third-order convergence: |e| < 2^-17 leaves
// ~1e-17); 1/w = y0^7 / (1 - e) ~ y0^7 (1 + e + e^2).
__device__ __forceinline__ void root7(double w, double& y, double& inv_w)
{
    const float q = log2_hi(w) * (-1.0f / 7.0f);
    const float qr = q + 12582912.0f;  // the nearest integer in the low mantissa bits
    const int n = __float_as_int(qr);
    const int f = __float_as_int(ex2_fast(q - (qr - 12582912.0f)));  // 2^[-1/2, 1/2]
    const double y0 = __hiloint2double((f >> 3) + ((1023 - 127) << 20) + ((n - 0x4b400000) << 20), f << 29);
    const double y2 = y0 * y0, y3 = y2 * y0, y6 = y3 * y3, y7 = y6 * y0;
    const double e = fma(-w, y7, 1.0);
    y = fma(y0, e * fma(e, 8.0 / 98.0, 1.0 / 7.0), y0);
    inv_w = fma(y7, fma(e, e, e), y7);
}

// b^7 = p_rr / p_L from the two-rarefaction estimate's base b (1/z = 7 to
// within 1e-14 on the fast path, which moves b^(1/z) by less than an ulp or
// two; the rounding of b alone moves b^7 by as much).  A negative base gives
// a negative result (the reference's pow gives NaN there); both make every
// "p_rr > p_K" test false, so the wave speeds agree.
__device__ __forceinline__ double pow7(double b)
{
    const double b2 = b * b, b3 = b2 * b, b6 = b3 * b3;
    return b6 * b;
}

// Velocities, pressure and 1/rho, and mn un (the advected normal momentum,
// shared by the kinetic energy and the flux): p = (gamma-1) E - (gamma-1)
// eps/2 (m . u).
template <int D, int DIR>
struct Prim {
    double ir, u[D], p, mnu;
    __device__ __forceinline__ Prim(const double (&U)[D + 2], const K<double>& k)
    {
        ir = rcp_fast(U[0]);
#pragma unroll
        for (int d = 0; d < D; ++d) u[d] = U[1 + d] * ir;
        mnu = U[1 + DIR] * u[DIR];
        double mu = mnu;
#pragma unroll
        for (int d = 0; d < D; ++d)
            if (d != DIR) mu = fma(U[1 + d], u[d], mu);
        p = fma(k.neg_gm1_heps, mu, k.gm1 * U[1 + D]);
    }
};

__device__ __forceinline__ bool both_zero(double a, double b)
{
    return (((unsigned)(__double2hiint(a) | __double2hiint(b)) << 1) | (unsigned)(__double2loint(a) | __double2loint(b))) == 0u;
}
__device__ __forceinline__ bool same_sign(double a, double b) { return (__double2hiint(a) ^ __double2hiint(b)) >= 0; }
__device__ __forceinline__ bool neg_bit(double a) { return __double2hiint(a) < 0; }
__device__ __forceinline__ bool at_least_one(double a) { return __double2hiint(a) >= 0x3ff00000; }

// A quarter of the limiter value of Flux_Helpers.cpp:103-111 and
// Limiters.H:29-73 without branches; sum = num + den.  With r = num / den
// every limiter is, for r > 0, a single quotient whose operands the case of
// r selects (minbee: num / den for r <= 1, 2 den / sum above; van Leer: 2
// min-side / sum; van Albada: num sum / (num^2 + den^2) for r <= 1, 2 den /
// sum above; superbee: 2 num / den, 1, 2 den / sum), so it takes one
// reciprocal; the cases are decided from num and den exactly (r > 1 is |num|
// > |den| with equal signs; the sign tests are integer ones).  Van Albada's
// squares leave the range for differences below 1e-154 or above 1e154, so
// a power of two brings the larger one to 1 .. 2 there (three products and
// integer selects: x and y sweeps of 2048^2 98 / 86 us without, 99 / 88 with, a
// branch around them 102 / 89).
template <int LIM>
__device__ __forceinline__ double quarter_limiter(double num, double den, double sum)
{
    if constexpr (LIM == LIM_VAN_ALBADA) {
        const int top = max(__double2hiint(num) & 0x7fffffff, __double2hiint(den) & 0x7fffffff);
        const bool inside = (unsigned)(top - ((1023 - 500) << 20)) <= (1000u << 20);
        const double s = __hiloint2double(inside ? 0x3ff00000 : 0x7fe00000 - min(top & 0x7ff00000, 0x7fd00000), 0);
        num *= s;
        den *= s;
        sum *= s;
    }
    const double an = fabs(num), ad = fabs(den);
    const bool big = an > ad;
    double phi;
    if constexpr (LIM == LIM_MINBEE) {
        const double q = (big ? den : num) * rcp_fast(big ? sum : den);
        phi = q * (big ? 0.5 : 0.25);
    } else if constexpr (LIM == LIM_VAN_LEER) {
        phi = 0.5 * (big ? den : num) * rcp_fast(sum);
    } else if constexpr (LIM == LIM_VAN_ALBADA) {
        const double q = (big ? den : num * sum) * rcp_fast(big ? sum : fma(num, num, den * den));
        phi = q * (big ? 0.5 : 0.25);
    } else {
        const bool half = 2.0 * an <= ad;
        const double q = 0.5 * (big ? den : num) * rcp_fast(big ? sum : den);
        phi = (half || big) ? q : 0.25;
    }
    phi = same_sign(num, den) ? phi : 0.0;
    return both_zero(num, den) ? 0.25 : phi;
}

// The half step of both reconstructed states by the difference of their
// physical fluxes (Flux_Helpers.cpp:123-148).
template <int D, int DIR>
__device__ __forceinline__ void half_step(double (&UL)[D + 2], double (&UR)[D + 2], const K<double>& k, double hdtdx)
{
    constexpr int NC = D + 2;
    constexpr int E = D + 1;
    const Prim<D, DIR> a(UL, k), b(UR, k);
    double dF[NC];
    dF[0] = UR[1 + DIR] - UL[1 + DIR];
#pragma unroll
    for (int d = 0; d < D; ++d)
        dF[1 + d] = d == DIR ? fma(b.p - a.p, k.inv_eps, b.mnu - a.mnu)
                             : fma(UR[1 + DIR], b.u[d], -(UL[1 + DIR] * a.u[d]));
    dF[E] = fma(UR[E] + b.p, b.u[DIR], -((UL[E] + a.p) * a.u[DIR]));
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        UL[n] = fma(-hdtdx, dF[n], UL[n]);
        UR[n] = fma(-hdtdx, dF[n], UR[n]);
    }
}

template <int D, int DIR, int LIM>
__device__ __forceinline__ void muscl_cell_f64(const double (&Um)[D + 2], const double (&U0)[D + 2], const double (&Up)[D + 2],
                                                const K<double>& k, double hdtdx, double (&UL)[D + 2], double (&UR)[D + 2])
{
    constexpr int NC = D + 2;
    constexpr int E = D + 1;
    // 0.5 phi delta with delta = 0.5 (U0 - Um) + 0.5 (Up - U0) written as
    // 0.25 phi (Up - Um) (within an ulp of the reference's rounding)
    double d2[NC];
#pragma unroll
    for (int n = 0; n < NC; ++n) d2[n] = Up[n] - Um[n];
    const double qphi = quarter_limiter<LIM>(U0[E] - Um[E], Up[E] - U0[E], d2[E]);
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        UL[n] = fma(-qphi, d2[n], U0[n]);
        UR[n] = fma(qphi, d2[n], U0[n]);
    }
    half_step<D, DIR>(UL, UR, k, hdtdx);
}

// quarter_limiter for a limiter known at run time: the same quotients, the
// operands selected (the limiter is uniform over the launch).  A limiter of
// differences so small (or large) that the reciprocal, which flushes subnormal
// operands, or van Albada's squares leave the range comes out as NaN; the cell
// stage sees that by one integer comparison and takes quarter_limiter_scaled
// instead.  Such differences are ordinary where a component is limited on its
// own ratio: ahead of a wave a transverse momentum falls by orders of magnitude
// per cell, down to the last subnormal.
__device__ __forceinline__ double quarter_limiter_rt(int lim, double num, double den, double sum)
{
    const double an = fabs(num), ad = fabs(den);
    const bool big = an > ad, leer = lim == LIM_VAN_LEER, albada = lim == LIM_VAN_ALBADA, bee = lim == LIM_SUPERBEE;
    const double top = big ? den : (albada ? num * sum : num);
    const double bottom = (big || leer) ? sum : (albada ? fma(num, num, den * den) : den);
    double phi = top * rcp_fast(bottom) * ((big || leer || bee) ? 0.5 : 0.25);
    phi = (bee && !big && 2.0 * an > ad) ? 0.25 : phi;
    phi = same_sign(num, den) ? phi : 0.0;
    return both_zero(num, den) ? 0.25 : phi;
}

// The high word of a limiter value, which tells NaN (and anything not in
// 0 .. 0.5) from the values there are.
__device__ __forceinline__ unsigned limiter_word(double q) { return (unsigned)__double2hiint(q); }
__device__ __forceinline__ bool limiter_failed(unsigned word) { return word > 0x3fe00000u; }

// The same limiter value with num and den brought to the size of one by a
// power of two (subnormal ones too): every limiter depends on their ratio
// alone.
__device__ __forceinline__ double quarter_limiter_scaled(int lim, double num, double den)
{
    const int top = max(__double2hiint(num) & 0x7fffffff, __double2hiint(den) & 0x7fffffff);
    const double s = __hiloint2double(0x7fe00000 - min(top & 0x7ff00000, 0x7fd00000), 0);
    num *= s;
    den *= s;
    return quarter_limiter_rt(lim, num, den, num + den);
}

// Cell stage of the general path (any limiting variables, muscl_cell above):
// one quotient per limiter value and the half step of the fast path.  One
// branch per cell for the limiters that left the range (gamma 5/3, each
// component on its own ratio, 192^3 x / y / z: 442 / 292 / 317 us without it,
// 441 / 301 / 326 now; a range test per limiter 477 / 315 / 340).
template <int D, int DIR>
__device__ __forceinline__ void muscl_cell_gen(const double (&Um)[D + 2], const double (&U0)[D + 2],
                                               const double (&Up)[D + 2], const K<double>& k, double hdtdx,
                                               double (&UL)[D + 2], double (&UR)[D + 2])
{
    constexpr int NC = D + 2;
    double qphi[NC];
    if (k.uniform_var >= 0) {
        const int v = k.uniform_var;
        const double m = sel(Um, v), c = sel(U0, v), p = sel(Up, v);
        double q = quarter_limiter_rt(k.limiter, c - m, p - c, p - m);
        if (limiter_failed(limiter_word(q))) q = quarter_limiter_scaled(k.limiter, c - m, p - c);
#pragma unroll
        for (int n = 0; n < NC; ++n) qphi[n] = q;
    } else {
        double num[NC], den[NC];
        unsigned worst = 0;
        if (!k.need_prim) {
#pragma unroll
            for (int n = 0; n < NC; ++n) {
                const int v = k.lim_var[n];
                const double m = v == n ? Um[n] : sel(Um, v), c = v == n ? U0[n] : sel(U0, v), p = v == n ? Up[n] : sel(Up, v);
                num[n] = c - m;
                den[n] = p - c;
            }
        } else {
            double Qm[NC], Q0[NC], Qp[NC];
            auto prim = [&](const double (&U)[NC], double (&q)[NC]) {
                const Prim<D, DIR> w(U, k);
                q[0] = U[0];
#pragma unroll
                for (int d = 0; d < D; ++d) q[1 + d] = w.u[d];
                q[1 + D] = w.p;
            };
            prim(Um, Qm);
            prim(U0, Q0);
            prim(Up, Qp);
#pragma unroll
            for (int n = 0; n < NC; ++n) {
                const int v = k.lim_var[n];
                const bool pr = k.lim_prim[n] != 0;
                const double m = pr ? sel(Qm, v) : sel(Um, v), c = pr ? sel(Q0, v) : sel(U0, v), p = pr ? sel(Qp, v) : sel(Up, v);
                num[n] = c - m;
                den[n] = p - c;
            }
        }
#pragma unroll
        for (int n = 0; n < NC; ++n) {
            qphi[n] = quarter_limiter_rt(k.limiter, num[n], den[n], num[n] + den[n]);
            worst = max(worst, limiter_word(qphi[n]));
        }
        if (limiter_failed(worst)) {
#pragma unroll
            for (int n = 0; n < NC; ++n)
                if (limiter_failed(limiter_word(qphi[n]))) qphi[n] = quarter_limiter_scaled(k.limiter, num[n], den[n]);
        }
    }
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const double d2 = Up[n] - Um[n];
        UL[n] = fma(-qphi[n], d2, U0[n]);
        UR[n] = fma(qphi[n], d2, U0[n]);
    }
    half_step<D, DIR>(UL, UR, k, hdtdx);
}

// The powers of the Toro estimate for any gamma: t = w^(-z), 1/w, and
// b^(1/z) (0 for b <= 0).  With 1/z = root_k to within 1e-12 (gamma = 7/5,
// 5/3, ...) the iteration of root7 for that k, and to first order the factors
// w^(1/k - z) = 1 + (1/k - z) ln w and b^(1/z - k) = 1 + (1/z - k) ln b;
// otherwise, or for extreme arguments, pow().
__device__ __forceinline__ double ipow(double y, int k)
{
    const double y2 = y * y, y4 = y2 * y2;
    if (k == 7) return y4 * y2 * y;
    if (k == 5) return y4 * y;
    double r = y;
    for (int i = 1; i < k; ++i) r *= y;
    return r;
}
__device__ __forceinline__ void root_gen(double w, const K<double>& c, double& t, double& inv_w)
{
    if (c.root_k == 0 || !(w > 1e-30 && w < 1e30)) {
        t = pow(w, c.neg_z);
        inv_w = 1.0 / w;
        return;
    }
    const float l2 = log2_hi(w);
    const float q = -l2 * (float)c.root_ik;
    const float qr = q + 12582912.0f;
    const int n = __float_as_int(qr);
    const int f = __float_as_int(ex2_fast(q - (qr - 12582912.0f)));
    const double y0 = __hiloint2double((f >> 3) + ((1023 - 127) << 20) + ((n - 0x4b400000) << 20), f << 29);
    const double yk = ipow(y0, c.root_k);
    const double e = fma(-w, yk, 1.0);
    t = fma(y0, fma(e, fma(e, c.root_c2, c.root_ik), c.root_dneg_l2 * (double)l2), y0);
    inv_w = fma(yk, fma(e, e, e), yk);
}
__device__ __forceinline__ double pow_ratio_gen(double b, const K<double>& c)
{
    if (!(b > 0.0)) return 0.0;
    if (c.root_k == 0 || !(b > 1e-30 && b < 1e30)) return pow(b, c.inv_z);
    const double bk = ipow(b, c.root_k);
    return fma(bk, c.root_dpos_l2 * (double)log2_hi(b), bk);
}

// HLLC (hllc_face above, HLLC.cpp:90-172 with HLLC.H:214-337), rearranged to
// spend fewer operations on the FP64 pipe, which bounds the sweeps:
//  * the two-rarefaction pressure as a ratio: p_rr / p_L = b^(1/z) with b =
//    (c_L + c_R - (gamma-1)/2 (u_R - u_L)) / (c_L + c_R (p_L/p_R)^z), so one
//    seventh root serves both sides, and p_rr / p_R = (p_rr / p_L)(p_L / p_R)
//    comes out of the same iteration;
//  * with a_K = c_K q_K > 0 the speeds are S_L = u_L - a_L, S_R = u_R + a_R,
//    and S* = ((p_L - p_R)/eps + m_L u_L + m_R u_R) / (m_L + m_R), m_K =
//    rho_K a_K;
//  * the star flux in advective form, with d_K = S_K - u_K = -a_L or a_R and
//    du = S* - u_K: rho* = rho_K d_K / (d_K - du), p* = p_K + eps rho_K d_K du,
//    E* = (E_K d_K + du (p_K + eps rho_K d_K S*)) / (d_K - du), F = S* (rho*,
//    rho* u*, E* + p*) + p*/eps.  With du = 0 the same expressions give rho_K,
//    p_K and E_K to within three roundings whatever the Mach number, so they
//    are the supersonic flux too.  (S_K - S* from the rounded S_K carries Mach x
//    2^-53 there: 1e-12 at Mach 1e4.  Selecting m_n and E_K instead costs the
//    registers of both sides: x sweep of 2048^2 108 us against 99.)
// GEN: any gamma, by root_gen / pow_ratio_gen.
template <int D, int DIR, bool GEN>
__device__ __forceinline__ void hllc_face_f64(const double (&L)[D + 2], const double (&R)[D + 2], const K<double>& k,
                                               double (&F)[D + 2])
{
    constexpr int E = D + 1;
    const Prim<D, DIR> l(L, k), r(R, k);
    // the estimate's clamped density and pressure (HLLC.H:255-260)
    const bool okL = L[0] >= kMinRho, okR = R[0] >= kMinRho;
    const double rhoL = okL ? L[0] : kMinRho, rhoR = okR ? R[0] : kMinRho;
    const double icL = okL ? l.ir : 1.0 / kMinRho, icR = okR ? r.ir : 1.0 / kMinRho;
    const double pL = l.p >= kMinP ? l.p : kMinP, pR = r.p >= kMinP ? r.p : kMinP;
    const double uL = l.u[DIR], uR = r.u[DIR];
    // positive arguments: p >= 1e-14 and 1 / rho <= 1e14 (clamped above)
    const double cL = sqrt_pos(k.gamma_inv_eps * pL * icL);
    const double cR = sqrt_pos(k.gamma_inv_eps * pR * icR);
    double t, p_lr;  // (p_L / p_R)^z and p_L / p_R
    if constexpr (GEN) root_gen(pR * rcp_fast(pL), k, t, p_lr);
    else root7(pR * rcp_fast(pL), t, p_lr);
    const double b = fma(-k.half_gm1, uR - uL, cL + cR) * rcp_fast(fma(cR, t, cL));
    const double rrL = GEN ? pow_ratio_gen(b, k) : pow7(b);
    const double rrR = rrL * p_lr;
    // q_K = sqrt(1 + (gamma+1)/(2 gamma) (max(p_rr / p_K, 1) - 1)): the select
    // is on the argument (whose value at 1 is exactly 1), since a select
    // between a root and 1 becomes a branch around the root
    const double aL = cL * sqrt_pos(fma(k.gp1_2g, at_least_one(rrL) ? rrL : 1.0, k.one_m_gp1_2g));
    const double aR = cR * sqrt_pos(fma(k.gp1_2g, at_least_one(rrR) ? rrR : 1.0, k.one_m_gp1_2g));
    const double SL = uL - aL, SR = uR + aR;
    const double mL = rhoL * aL, mR = rhoR * aR;
    const double Ss = fma(mL, uL, fma(mR, uR, (pL - pR) * k.inv_eps)) * rcp_fast(mL + mR);

    // left states when S_L >= 0 or S* >= 0, right ones otherwise; supersonic
    // when S_L >= 0 or S_R < 0 (sign bits)
    const bool useL = !(neg_bit(SL) && neg_bit(Ss));
    const bool star = useL ? neg_bit(SL) : !neg_bit(SR);
    const double un = useL ? uL : uR, p = useL ? l.p : r.p, en = useL ? L[E] : R[E];
    const double dK = useL ? -aL : aR;
    const double us = star ? Ss : un;
    const double m = (useL ? L[0] : R[0]) * dK;
    const double du = us - un;
    const double rb = rcp_fast(dK - du);
    const double me = m * k.eps;
    const double ps = fma(me, du, p);
    const double es = fma(du, fma(me, us, p), en * dK) * rb;
    const double mass = m * rb * us;
    F[0] = mass;
#pragma unroll
    for (int d = 0; d < D; ++d)
        F[1 + d] = d == DIR ? fma(mass, us, ps * k.inv_eps) : mass * (useL ? l.u[d] : r.u[d]);
    F[E] = us * (es + ps);
}

// |u| + c, within a few ulp; NaN for a negative pressure or density, as the
// roots are, and infinite where a square is.  Both radicands are offset by 1e-300: exact for every normal
// value above 1e-284, and a fluid at rest (or without pressure) adds 1e-150
// instead of 0, which the sum's rounding drops unless both vanish (reduce_ws
// takes such a maximum back to 0).
template <int D>
__device__ __forceinline__ double wave_speed_f64(const double (&U)[D + 2], const K<double>& k)
{
    const Prim<D, 0> q(U, k);
    double mu = q.mnu;
#pragma unroll
    for (int d = 1; d < D; ++d) mu = fma(U[1 + d], q.u[d], mu);
    const double c2 = fma(k.gamma_inv_eps * q.p, q.ir, 1e-300), v2 = fma(mu, q.ir, 1e-300);
    auto root = [](double x) {
        const double r = sqrt_pos(x);
        return __double2hiint(x) == 0x7ff00000 ? x : r;  // (the maximum keeps an infinity)
    };
    return root(c2) + root(v2);
}

// ---- FP32 storage: the same scheme with the hardware approximations -------

// x^(-z) (HLLC.H:272) and 1/x on the special-function unit.
__device__ __forceinline__ void root7_neg_z_f32(float x, const K<float>& c, float& y, float& inv_x)
{
    y = ex2_fast(c.neg_z * lg2_fast(x));
    inv_x = rcp_fast(x);
}

template <int D>
__device__ __forceinline__ void to_prim_f32(const float (&U)[D + 2], const K<float>& k, float (&q)[D + 2], float& inv_rho)
{
    inv_rho = rcp_fast(U[0]);
    q[0] = U[0];
#pragma unroll
    for (int d = 0; d < D; ++d) q[1 + d] = U[1 + d] * inv_rho;
    float usq = q[1] * q[1];
#pragma unroll
    for (int d = 1; d < D; ++d) usq = usq + q[1 + d] * q[1 + d];
    q[1 + D] = k.gm1 * (U[1 + D] - k.half_eps * U[0] * usq);
}

template <int D, int DIR>
__device__ __forceinline__ void phys_flux_f32(const float (&U)[D + 2], const K<float>& k, float (&F)[D + 2])
{
    float q[D + 2], ir;
    to_prim_f32<D>(U, k, q, ir);
    phys_flux<float, D, DIR>(U, q, k, F);
}

// The limiter value of Flux_Helpers.cpp:103-111 and Limiters.H:29-73 without
// branches.  With r = num / den, minbee, van Leer and superbee are, for
// r > 0, a single quotient of num and den whose operands the case of r
// selects (minbee: num / den for r <= 1, 2 den / (den + num) above; van
// Leer: 2 min-side / (den + num); superbee: 2 num / den, 1, 2 den / (den +
// num)), so they take one reciprocal; the cases are decided from num and den
// exactly (r > 1 is |num| > |den| with equal signs), which agrees with the
// rounded quotient except where that rounds to exactly 1 or 1/2, and there
// both formulas give the same value to an ulp.
template <int LIM>
__device__ __forceinline__ float limiter_value_f32(float num, float den)
{
    const bool pos = (num > 0.0f && den > 0.0f) || (num < 0.0f && den < 0.0f);  // r > 0
    const float an = fabs(num), ad = fabs(den);
    float phi;
    if constexpr (LIM == LIM_MINBEE) {
        const bool big = an > ad;  // r > 1
        phi = (big ? 2.0f * den : num) * rcp_fast(big ? den + num : den);
    } else if constexpr (LIM == LIM_VAN_LEER) {
        // 2 r / (1 + r) for r <= 1, 2 / (1 + r) above
        phi = 2.0f * (an > ad ? den : num) * rcp_fast(den + num);
    } else if constexpr (LIM == LIM_VAN_ALBADA) {
        const float r = num * rcp_fast(den);
        phi = fmin(r * (1.0f + r) * rcp_fast(1.0f + r * r), 2.0f * rcp_fast(1.0f + r));
    } else {
        // 2 r for r <= 1/2, 1 for r <= 1, min(r, 2 / (1 + r), 2) = 2 / (1 + r) above
        const bool big = an > ad, half = 2.0f * an <= ad;
        const float q = (big ? 2.0f * den : 2.0f * num) * rcp_fast(big ? den + num : den);
        phi = (half || big) ? q : 1.0f;
    }
    phi = pos ? phi : 0.0f;
    return (num == 0.0f && den == 0.0f) ? 1.0f : phi;
}

template <int D, int DIR, int LIM>
__device__ __forceinline__ void muscl_cell_f32(const float (&Um)[D + 2], const float (&U0)[D + 2], const float (&Up)[D + 2],
                                                const K<float>& k, float hdtdx, float (&UL)[D + 2], float (&UR)[D + 2])
{
    constexpr int NC = D + 2;
    constexpr int E = D + 1;
    // 0.5 phi delta with delta = 0.5 (U0 - Um) + 0.5 (Up - U0) written as
    // 0.25 phi (Up - Um) (within an ulp of the reference's rounding)
    const float qphi = 0.25f * limiter_value_f32<LIM>(U0[E] - Um[E], Up[E] - U0[E]);
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const float d2 = Up[n] - Um[n];
        UL[n] = fma(-qphi, d2, U0[n]);
        UR[n] = fma(qphi, d2, U0[n]);
    }
    float FL[NC], FR[NC];
    phys_flux_f32<D, DIR>(UL, k, FL);
    phys_flux_f32<D, DIR>(UR, k, FR);
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        const float dF = hdtdx * (FR[n] - FL[n]);
        UL[n] -= dF;
        UR[n] -= dF;
    }
}

template <int D, int DIR>
__device__ __forceinline__ void hllc_face_f32(const float (&L)[D + 2], const float (&R)[D + 2], const K<float>& k,
                                               float (&F)[D + 2])
{
    constexpr int NC = D + 2;
    float qL[NC], qR[NC], irL, irR;
    to_prim_f32<D>(L, k, qL, irL);
    to_prim_f32<D>(R, k, qR, irR);
    const float rhoL = fmax(qL[0], (float)kMinRho), rhoR = fmax(qR[0], (float)kMinRho);
    const float pL = fmax(qL[1 + D], (float)kMinP), pR = fmax(qR[1 + D], (float)kMinP);
    const float uL = qL[1 + DIR], uR = qR[1 + DIR];
    const float icL = (qL[0] >= (float)kMinRho) ? irL : (float)(1.0 / kMinRho);
    const float icR = (qR[0] >= (float)kMinRho) ? irR : (float)(1.0 / kMinRho);
    // positive arguments: p >= 1e-14 and 1 / rho <= 1e14 (clamped above),
    // and 1 + (gamma+1)/(2 gamma) (p_rr / p - 1) > 1 under p_rr > p
    const float cL = sqrt_fast(k.gamma_inv_eps * pL * icL);
    const float cR = sqrt_fast(k.gamma_inv_eps * pR * icR);
    float yL, yR, ipL, ipR;
    root7_neg_z_f32(pL, k, yL, ipL);
    root7_neg_z_f32(pR, k, yR, ipR);
    const float base = (cL + cR - k.half_gm1 * (uR - uL)) * rcp_fast(cL * yL + cR * yR);
    const float p_rr = ex2_fast(k.inv_z * lg2_fast(base));  // NaN for a negative base, as the reference's pow
    const float qwL = (p_rr > pL) ? sqrt_fast(1.0f + k.gp1_2g * (p_rr * ipL - 1.0f)) : 1.0f;
    const float qwR = (p_rr > pR) ? sqrt_fast(1.0f + k.gp1_2g * (p_rr * ipR - 1.0f)) : 1.0f;
    const float SL = uL - cL * qwL;
    const float SR = uR + cR * qwR;
    const float dL = SL - uL, dR = SR - uR;
    const float denom = rhoL * dL - rhoR * dR;
    const float Ss_raw = ((pR - pL) * k.inv_eps + rhoL * uL * dL - rhoR * uR * dR) * rcp_fast(denom);
    const float Ss = (denom != 0.0f) ? Ss_raw : 0.0f;

    const bool useL = (SL >= 0.0f) || (Ss >= 0.0f);
    const bool star = useL ? (SL < 0.0f) : (SR >= 0.0f);
    float UK[NC], qK[NC];
#pragma unroll
    for (int n = 0; n < NC; ++n) {
        UK[n] = useL ? L[n] : R[n];
        qK[n] = useL ? qL[n] : qR[n];
    }
    const float irK = useL ? irL : irR;
    const float SK = useL ? SL : SR;
    phys_flux<float, D, DIR>(UK, qK, k, F);
    // star state (HLLC.H:311-337): with m = rho_K (S_K - u_K), b = S_K - S*,
    // scale = m / b = m^2 / (m b) and p_K / m = p_K b / (m b)
    const float rhoK = qK[0], uK = qK[1 + DIR], pK = qK[1 + D];
    const float m = rhoK * (SK - uK);
    const float bq = SK - Ss;
    const float rmb = rcp_fast(m * bq);
    const float scale = m * m * rmb;
    const float eterm = UK[1 + D] * irK + (Ss - uK) * (Ss * k.eps + pK * bq * rmb);
    F[0] = star ? F[0] + SK * (scale - UK[0]) : F[0];
#pragma unroll
    for (int d = 0; d < D; ++d) {
        const float s = (d == DIR) ? Ss : qK[1 + d];
        F[1 + d] = star ? F[1 + d] + SK * (s * scale - UK[1 + d]) : F[1 + d];
    }
    F[1 + D] = star ? F[1 + D] + SK * (eterm * scale - UK[1 + D]) : F[1 + D];
}

template <int D>
__device__ __forceinline__ float wave_speed_f32(const float (&U)[D + 2], const K<float>& k)
{
    float q[D + 2], ir;
    to_prim_f32<D>(U, k, q, ir);
    float vsq = q[1] * q[1];
#pragma unroll
    for (int d = 1; d < D; ++d) vsq = vsq + q[1 + d] * q[1 + d];
    return sqrt_fast(k.gamma_inv_eps * q[1 + D] * ir) + sqrt_fast(vsq);
}

// Method dispatch: cell stage (reconstruction + half step for MUSCL-Hancock
// and SLIC; identity for first-order methods) and face stage.  LIM >= 0
// selects the fast path (MUSCL-Hancock only) with that compile-time limiter;
// LIM = -1 is the general path (runtime limiter and limiting variables, any
// gamma).
template <typename T, int D, int DIR, int METHOD, int LIM = -1>
struct Scheme {
    static constexpr int NC = D + 2;
    static constexpr bool kReconstruct = (METHOD == M_MUSCL || METHOD == M_SLIC);
    static constexpr bool kFast = (LIM >= 0);
    static constexpr int kHalo = kReconstruct ? 2 : 1;
    static_assert(!kFast || METHOD == M_MUSCL, "the fast path is MUSCL-Hancock only");

    __device__ __forceinline__ static void cell(const T (&Um)[NC], const T (&U0)[NC], const T (&Up)[NC],
                                                const K<T>& k, T hdtdx, T (&UL)[NC], T (&UR)[NC])
    {
        if constexpr (kFast) {
            constexpr int L = LIM < 0 ? 0 : LIM;
            if constexpr (sizeof(T) == 8) muscl_cell_f64<D, DIR, L>(Um, U0, Up, k, hdtdx, UL, UR);
            else muscl_cell_f32<D, DIR, L>(Um, U0, Up, k, hdtdx, UL, UR);
        } else if constexpr (kReconstruct) {
            if constexpr (sizeof(T) == 8) muscl_cell_gen<D, DIR>(Um, U0, Up, k, hdtdx, UL, UR);
            else muscl_cell<T, D, DIR>(Um, U0, Up, k, hdtdx, UL, UR);
        } else {
#pragma unroll
            for (int n = 0; n < NC; ++n) UL[n] = UR[n] = U0[n];
        }
    }

    // L: state left of the face (UR of the left cell), R: state right of it.
    __device__ __forceinline__ static void face(const T (&L)[NC], const T (&R)[NC], const K<T>& k, T half_dx_dt,
                                                T dt_2dx, T (&F)[NC])
    {
        if constexpr (kFast) {
            if constexpr (sizeof(T) == 8) hllc_face_f64<D, DIR, false>(L, R, k, F);
            else hllc_face_f32<D, DIR>(L, R, k, F);
        } else if constexpr (METHOD == M_MUSCL || METHOD == M_HLLC) {
            if constexpr (sizeof(T) == 8) hllc_face_f64<D, DIR, true>(L, R, k, F);
            else hllc_face<T, D, DIR>(L, R, k, F);
        } else if constexpr (METHOD == M_SLIC || METHOD == M_FORCE) {
            force_face<T, D, DIR>(L, R, k, half_dx_dt, dt_2dx, F);
        } else {
            lf_face<T, D, DIR>(L, R, k, half_dx_dt, F);
        }
    }

    __device__ __forceinline__ static T speed(const T (&U)[NC], const K<T>& k)
    {
        if constexpr (!kFast) return wave_speed<T, D>(U, k);
        else if constexpr (sizeof(T) == 8) return wave_speed_f64<D>(U, k);
        else return wave_speed_f32<D>(U, k);
    }
};

}  // namespace bamrex
