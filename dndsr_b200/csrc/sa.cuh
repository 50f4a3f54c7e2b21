// Spalart-Allmaras model terms of the NS_SA model (6 conservative variables, the sixth being
// rho nuTilde / muRef): eddy viscosity, the nuTilde diffusion flux, the passive-scalar upwind flux
// and the source term with its diagonal Jacobian.  Settings are the reference defaults (SADESMode
// 1 IDDES shielding, rotation correction on, SAVersion 0) and its compiled options (negative-SA
// model, ft2 term).  The state-dependent routines are templated on the scalar type: real for the
// residual, dual numbers for its derivatives.
#pragma once
#include "solver.cuh"
#include "dual.cuh"

namespace dndsb
{
struct SAConst
{
    static constexpr real cb1 = 0.1355, cb2 = 0.622, sigma = 2.0 / 3.0, cnu1 = 7.1, cnu2 = 0.7, cnu3 = 0.9, cw2 = 0.3, cw3 = 2,
                          kappa = 0.41, rlim = 10, cn1 = 16.0, ct3 = 1.2, ct4 = 0.5;
};

// EulerEvaluator.hpp:791-833 getMuTur (chi smoothed below 10 by the negative-SA model)
template <typename T>
DNDSB_HD T sa_mu_tur(const T *U, real muRef, const T &muf)
{
    T Chi = U[5] * muRef / muf;
    if (Chi < 10)
        Chi = 0.05 * log(1 + exp(20 * Chi));
    T Chi3 = Chi * Chi * Chi;
    T fnu1 = Chi3 / (Chi3 + SAConst::cnu1 * SAConst::cnu1 * SAConst::cnu1);
    return muf * dmax(Chi * fnu1, 0.0);
}

// EulerEvaluator.hpp:835-877 visFluxTurVariable: the nuTilde diffusion flux through n (GP is the
// primitive gradient [3][6], the sixth column d(U5 / rho))
template <typename T>
DNDSB_HD T sa_diffusion_flux(const T *U, const T *GP, const real *n, real muRef, const T &mufPhy)
{
    T fn = 1;
    if (U[5] < 0)
    {
        T Chi = U[5] * muRef / mufPhy;
        fn = (SAConst::cn1 + Chi * Chi * Chi) / (SAConst::cn1 - Chi * Chi * Chi);
    }
    return (GP[0 * 6 + 5] * n[0] + GP[1 * 6 + 5] * n[1] + GP[2 * 6 + 5] * n[2]) * (mufPhy + U[5] * muRef * fn) / SAConst::sigma;
}

// EulerEvaluator_EvaluateDt.hxx:1413-1425: upwind flux of the SA variable with the Riemann
// solver's lam123 as dissipation speed (ransEigScheme 0)
template <typename T>
DNDSB_HD T sa_convective_flux(const T *UL, const T *UR, const real *n, const T &lam123)
{
    T vnL = (UL[1] * n[0] + UL[2] * n[1] + UL[3] * n[2]) / UL[0];
    T vnR = (UR[1] * n[0] + UR[2] * n[1] + UR[3] * n[2]) / UR[0];
    return ((vnL * UL[5] + vnR * UR[5]) - (UR[5] - UL[5]) * lam123) * 0.5;
}

constexpr real kSAFarDistance = 2.5873402367724347e33; // kVeryLarge^(1/6), the largest wall distance taken

template <typename T>
DNDSB_HD T sa_cube(const T &x) { return x * x * x; }
// x^(1/6) of x >= 0 (zero derivative at 0, as the power has in dual numbers)
DNDSB_HD real sa_root6(real x) { return sqrt(cbrt(x)); }
template <int N>
DNDSB_HD Dual<N> sa_root6(const Dual<N> &x)
{
    Dual<N> r;
    r.v = sa_root6(x.v);
    const real s = x.v != 0 ? r.v / (6 * x.v) : 0.0;
    for (int i = 0; i < N; i++)
        r.d[i] = s * x.d[i];
    return r;
}

// The state enters the source through rho, U5, mu and five invariants of the conservative gradient G [3][6]
template <typename T>
struct SAInvariants
{
    T ir, velo[3], nuh;                 // 1 / rho, velocity, nuTilde
    T dRho[3], dNu[3], dV[3][3];        // gradients of rho, nuTilde and the velocity (dV[i][j] = d v_j / d x_i)
    T om2, ss2, du2, dd, nn;            // vorticity, strain and gradient norms squared; dRho.dNu, dNu.dNu
};

template <typename T>
DNDSB_HD void sa_invariants(const T *U, const T *G, real muRef, SAInvariants<T> &q)
{
    q.ir = 1.0 / U[0];
    q.nuh = U[5] * muRef * q.ir;
    for (int j = 0; j < 3; j++)
        q.velo[j] = U[1 + j] * q.ir;
    for (int i = 0; i < 3; i++)
    {
        q.dRho[i] = G[i * 6 + 0];
        q.dNu[i] = (G[i * 6 + 5] * muRef - q.nuh * q.dRho[i]) * q.ir;
        for (int j = 0; j < 3; j++)
            q.dV[i][j] = (G[i * 6 + 1 + j] - q.dRho[i] * q.velo[j]) * q.ir;
    }
    q.om2 = q.ss2 = q.du2 = 0;
    for (int i = 0; i < 3; i++)
        for (int j = 0; j < 3; j++)
        {
            T o = 0.5 * (q.dV[j][i] - q.dV[i][j]);
            T sij = q.dV[i][j] + q.dV[j][i];
            q.om2 += o * o, q.ss2 += sij * sij, q.du2 += q.dV[i][j] * q.dV[i][j];
        }
    q.dd = q.dRho[0] * q.dNu[0] + q.dRho[1] * q.dNu[1] + q.dRho[2] * q.dNu[2];
    q.nn = q.dNu[0] * q.dNu[0] + q.dNu[1] * q.dNu[1] + q.dNu[2] * q.dNu[2];
}

// RANS_ke.hpp:985-1195 GetSource_SA: production P, destruction D and the diffusion factor fn, from
// (rho, U5, mu; S, SS, |grad v|).  Bound by the FP64 elementary functions, so whole powers are products, the sixth
// root is a square root of a cube root, and where a blending factor is exactly 0 or 1 (fe1 <= 1, fB = 1: next to the
// wall) the functions that it multiplies away are not evaluated.
template <typename T>
DNDSB_HD void sa_core(const T &rho, const T &n5, const T &mufPhy, const T &S, const T &SS, const T &diffUNorm, real muRef, real d, real lLES,
                      real hMax, T &P, T &D, T &fn)
{
    using C = SAConst;
    const real cw1 = C::cb1 / (C::kappa * C::kappa) + (1 + C::cb2) / C::sigma;
    const real k2 = C::kappa * C::kappa;
    const T ir = 1.0 / rho;
    T nuh = n5 * muRef * ir;
    T Chi = n5 * muRef / mufPhy;
    T Chi3 = sa_cube(Chi);
    T fnu1 = Chi3 / (Chi3 + C::cnu1 * C::cnu1 * C::cnu1);
    T fnu2 = 1 - Chi / (1 + Chi * fnu1);
    T SRotCor = 2.0 * dmin(0.0, S - SS);
    T ft2 = C::ct3 * exp(-C::ct4 * Chi * Chi);
    // the IDDES blend of the RANS and LES lengths (SADESMode 1)
    const real lRANS = d;
    T nufPhy = mufPhy * ir;
    T nuTur = nufPhy * dmax(Chi * fnu1, 0.0);
    T iden = 1.0 / (k2 * d * d * dmax(kSmall, diffUNorm));
    T psiSqr = Chi <= 0 ? T(100.0) : dmin(100.0, (1 - C::cb1 / (cw1 * k2 * 0.424) * (ft2 + (1 - ft2) * fnu2)) / (fnu1 * dmax(kSmall, 1 - ft2)));
    T psi = sqrt(dmax(psiSqr, 1.0));
    const real alphaIDDES = 0.25 - d / hMax;
    const real fB = dmin(2 * exp(-9. * alphaIDDES * alphaIDDES), 1.0);
    const real cl = 3.55, ct = 1.63;
    T rdt = nuTur * iden, rdl = nufPhy * iden;
    const real fe1 = 2. * exp(-(alphaIDDES >= 0 ? 11.09 : 9.0) * alphaIDDES * alphaIDDES);
    T fe = 0.0;
    if (fe1 > 1)
    {
        T ft = tanh(sa_cube(T(ct * ct * rdt)));
        T flt = (cl * cl * rdl) * (cl * cl * rdl);
        T fl = tanh((flt * flt) * (flt * flt) * flt);
        fe = (fe1 - 1.) * psi * (1. - dmax(ft, fl));
    }
    T dL = (1 + fe) * lRANS;
    if (fB < 1)
    {
        T fdTilde = dmax(fB, tanh(sa_cube(T(8 * rdt))));
        dL = fdTilde * dL + (1 - fdTilde) * lLES * psi;
    }
    dL = dmax(lLES * kSmall, dL);
    T idL = 1.0 / dL;
    T nd = nuh * idL; // nuTilde / d
    T Sbar = nuh / (k2 * dL * dL) * fnu2;
    T Sh = Sbar < -C::cnu2 * S ? T(S + S * (C::cnu2 * C::cnu2 * S + C::cnu3 * Sbar) / ((C::cnu3 - 2 * C::cnu2) * S - Sbar)) : T(S + Sbar);
    if (n5 < 0)
    {
        T Chi_3 = Chi3;
        fn = (C::cn1 + Chi_3) / (C::cn1 - Chi_3);
        D = -cw1 * nd * nd;
        P = C::cb1 * (1 - C::ct3) * fabs(S + SRotCor) * nuh;
        return;
    }
    T r = dmin(nuh / (Sh * (C::kappa * dL) * (C::kappa * dL) + kVerySmall), C::rlim);
    T g = r + C::cw2 * (sa_cube(T(r * r)) - r);
    const real cw36 = C::cw3 * C::cw3 * C::cw3 * C::cw3 * C::cw3 * C::cw3;
    T fw = g * sa_root6(T((1 + cw36) / (sa_cube(T(g * g)) + cw36)));
    fn = 1.0;
    D = (cw1 * fw - C::cb1 / k2 * ft2) * nd * nd;
    P = C::cb1 * (1 - ft2) * (Sh + SRotCor) * nuh;
}

// the source of the SA equation (mode 0 of GetSource_SA); with J (real only) its diagonal Jacobian (mode 1)
template <typename T>
DNDSB_HD T sa_source(const T *U, const T *G, real muRef, const T &mufPhy, real d, real lLES, real hMax, real *J = nullptr)
{
    using C = SAConst;
    SAInvariants<T> q;
    sa_invariants(U, G, muRef, q);
    T P, D, fn;
    sa_core(U[0], U[5], mufPhy, T(sqrt(q.om2) * sqrt(2.0)), T(sqrt(q.ss2) * (1. / sqrt(2.0))), T(sqrt(q.du2)), muRef, d, lLES, hMax, P, D, fn);
    if (J)
        *J = -dmin(value_of(U[0]) * (dmin(value_of(P), 0.0) * 1 - value_of(D) * 2) / muRef / (::fabs(value_of(U[5])) + kVerySmall), -kVerySmall);
    return U[0] * (P - D + q.nn * C::cb2 / C::sigma) / muRef - (U[5] * fn * muRef + mufPhy) * q.ir / C::sigma * q.dd / muRef;
}
// fluxFace viscous part at one point (EvaluateDt.hxx:1167-1209): laminar plus, for the SA model,
// mu_t (with Pr_t = 0.9 heat conduction) and the nuTilde diffusion flux
template <int NV, typename T>
DNDSB_D void point_viscous_flux(const EulerSettingsD &s, const T *UM, const T *GP, const real *n, bool adiabatic, T *Fv)
{
    const real gamma = s.gamma, cp = s.Rgas * gamma / (gamma - 1);
    T pM, a2M, HM;
    gas_thermal(UM[4], UM[0], T((UM[1] * UM[1] + UM[2] * UM[2] + UM[3] * UM[3]) / (UM[0] * UM[0])), gamma, pM, a2M, HM);
    T Tm = pM / ((gamma - 1) / gamma * cp * UM[0]);
    T mu = mu_eff(s.muModel, s.muGas, s.TRef, s.CSutherland, UM[0], Tm);
    if (NV == 6)
    {
        T muTur = sa_mu_tur(UM, s.muGas, mu);
        viscous_flux<NV>(UM, GP, n, adiabatic, gamma, mu + muTur, cp * muTur / 0.9 + cp * mu / s.prGas, cp, Fv);
        Fv[NV - 1] = sa_diffusion_flux(UM, GP, n, s.muGas, mu);
    }
    else
        viscous_flux<NV>(UM, GP, n, adiabatic, gamma, mu, cp * mu / s.prGas, cp, Fv);
}
} // namespace dndsb
