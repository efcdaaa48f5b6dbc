// fv_adjoint.cuh -- reverse mode (vector-Jacobian product) of the FP64 RHS, sm_100a.
//
// Given a residual weight Fbar (one row per cell, read on owned cells), the VJP accumulates
// Ubar += (dF/dU)^T Fbar for every cell, boundary ghosts and halos included. It is the exact
// transpose of the tangent the dual-number kernels propagate (the derivative of the branch the primal
// evaluation takes at limiter minima, flux-splitting switches and mass-fraction clips).
//
// Of the forward pass only per-cell data is kept: the limited gradients and aux gradients one RHS
// keeps anyway, plus the unlimited gradient, the limiter factor and the minimising face per component.
// Every per-face intermediate (face states, EOS decode, flux calculator) is recomputed:
//   k_gradient          forward gradients, with the limiter records
//   k_tile_adjoint      one CTA per tile. Per face: recompute the face states, the EOS decode and the flux
//                       calculator, then run the flux backwards into the face's shared-memory record.
//                       Per tile cell: sum the adjoints of its state, limited gradient, aux and aux
//                       gradient from its faces' records, then run the limiter and the least-squares
//                       gradient backwards from the records of the forward gradient pass.
//   k_adjoint_nonowned  the same cell step for boundary ghosts and halos, from per-face records.
//   k_adjoint_gather    per cell: the neighbour terms of the gradient, limiter and aux-gradient adjoints
//                       (a gather over the cell's faces, the transpose of the forward gathers), then the
//                       aux (T, u, Y) chain rule, added into Ubar.
//
// Reference functions reversed: CellInterpolant::ComputeFieldGradients and the limiter
// (src/finiteVolume/cellInterpolant.cpp:282-497), ComputeFluxSourceTerms and ProjectToFace (:499-639,
// :890-950), NavierStokesTransport::AdvectionFlux / DiffusionFlux (navierStokesTransport.cpp:99-207,
// 454-532), SpeciesTransport fluxes (speciesTransport.cpp:112-341), the flux calculators
// (ausm.cpp:2-43, ausmpUp.cpp:5-96, riemann.cpp / riemannSolver.cpp), PerfectGas and TChem decode.
#pragma once
#include "fv_kernels.cuh"

namespace abl {

// ---------------------------------------------------------------------------------------------------
// EOS pieces
// ---------------------------------------------------------------------------------------------------
// e = U1/rho - |rho u|^2 / (2 rho^2)
template <int DIM>
ABL_HD void internal_energy_vjp(const double* U, double eb, double* Ub) {
    const double irho = rcp64(U[0]);
    double vu = 0;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        const double vel = U[2 + d] * irho;
        Ub[2 + d] -= eb * vel * irho;
        vu += vel * U[2 + d];
    }
    Ub[1] += eb * irho;
    Ub[0] -= eb * (U[1] - vu) * irho * irho;
}

// reverse of fill_y (clip to [0, 1], renormalise or close with the last species)
template <int NSMAX>
ABL_HD void fill_y_vjp(int ns, double rho, const double* rhoY, const double* ysb, double* rhob, double* rhoYb) {
    const double irho = rcp64(rho);
    double y[NSMAX > 0 ? NSMAX : 1];
    bool act[NSMAX > 0 ? NSMAX : 1];
    double sum = 0.0;
ABL_UNROLL_SPECIES
    for (int s = 0; s < ns - 1; s++) {
        const double raw = rhoY[s] * irho;
        act[s] = raw > 0.0 && !(1.0 < raw);
        y[s] = pmin(1.0, pmax(0.0, raw));
        sum += y[s];
    }
    double irhob = 0.0, dot = 0.0;
    if (sum > 1.0) {
ABL_UNROLL_SPECIES
        for (int s = 0; s < ns - 1; s++) dot += ysb[s] * y[s];
    }
ABL_UNROLL_SPECIES
    for (int s = 0; s < ns - 1; s++) {
        double yb = sum > 1.0 ? ysb[s] / sum - dot / (sum * sum) : ysb[s] - ysb[ns - 1];
        if (!act[s]) yb = 0.0;
        rhoYb[s] += yb * irho;
        irhob += yb * rhoY[s];
    }
    *rhob -= irhob * irho * irho;
}

// reverse of the mixture temperature T(e_ref, Y) (implicit function of e_s(T, Y) = e_ref)
template <int DIM, int NSMAX>
ABL_HD void nasa_temperature_vjp(const Phys& P, int ns, const double* U, const double* ys, double T, double Tb, double* ysb, double* Ub) {
    double cv = 0, ek[NSMAX > 0 ? NSMAX : 1];
ABL_UNROLL_SPECIES
    for (int k = 0; k < ns; k++) {
        double c[6];
        species_poly(P, k, T, c);
        cv += ys[k] * poly_cv(c, T);
        ek[k] = poly_e(c, T);
    }
    const double q = Tb / cv;
ABL_UNROLL_SPECIES
    for (int k = 0; k < ns; k++) ysb[k] -= q * ek[k];
    internal_energy_vjp<DIM>(U, q, Ub);
}

// reverse of decode(): adjoints of the decoded e, a, p into the face state U
template <int DIM, int NSMAX>
ABL_HD void decode_vjp(const Phys& P, int ns, const double* U, const Decoded<double>& dd, double eb, double ab, double pb, double* Ub) {
    const double rho = U[0];
    if (NSMAX == 0 || P.eos == ABL_EOS_PERFECT_GAS) {
        double Tb = eb * P.cv + pb * P.r_gas * rho;
        if (dd.a > 0) Tb += ab * P.gamma * P.r_gas / (2.0 * dd.a);
        Ub[0] += pb * P.r_gas * dd.T;
        internal_energy_vjp<DIM>(U, Tb * P.icv, Ub);
        return;
    }
    constexpr int NY = NSMAX > 0 ? NSMAX : 1;
    double ys[NY], ysb[NY];
    fill_y(ns, rho, U + 2 + DIM, ys);
    const double T = dd.T;
    // one pass over the species at T: e_k and c_v,k serve the energy, the sound speed and the temperature's
    // own reverse (e_s(T, Y) = e_ref)
    double cv = 0, iw = 0, dcv = 0, ek[NY], ck[NY];
ABL_UNROLL_SPECIES
    for (int k = 0; k < ns; k++) {
        double c[6];
        species_poly(P, k, T, c);
        ek[k] = poly_e(c, T);
        ck[k] = poly_cv(c, T);
        cv += ys[k] * ck[k];
        dcv += ys[k] * poly_dcv(c, T);
        iw += ys[k] * P.inv_mw[k];
    }
    const double R = kRuniv * iw, icv = rcp64(cv);
    const double gamma = (cv + R) * icv;
    const double q = dd.a > 0 ? ab / (2.0 * dd.a) : 0.0;  // a = sqrt(gamma R T), gamma = 1 + R / cv
    const double gb = q * R * T;
    const double cvb = -gb * R * icv * icv;
    const double Rb = q * gamma * T + pb * rho * T + gb * icv;
    // e = e_s(T, Y): de/dT = cv, de/dY_k = e_k
    const double Tb = q * gamma * R + pb * rho * R + cvb * dcv + eb * cv;
    Ub[0] += pb * R * T;
    const double qT = Tb * icv;
ABL_UNROLL_SPECIES
    for (int k = 0; k < ns; k++) ysb[k] = (eb - qT) * ek[k] + cvb * ck[k] + Rb * kRuniv * P.inv_mw[k];
    internal_energy_vjp<DIM>(U, qT, Ub);
    fill_y_vjp<NSMAX>(ns, rho, U + 2 + DIM, ysb, Ub, Ub + 2 + DIM);
}

// reverse of cp_at (conductivity of Sutherland / constant-Lewis transport)
template <int DIM, int NSMAX>
ABL_HD void cp_at_vjp(const Phys& P, int ns, const double* U, double T, double cpb, double* Ub, double* Tb) {
    if (NSMAX == 0 || P.eos == ABL_EOS_PERFECT_GAS) return;
    constexpr int NY = NSMAX > 0 ? NSMAX : 1;
    double ys[NY], ysb[NY];
    fill_y(ns, U[0], U + 2 + DIM, ys);
    double dcv = 0;
ABL_UNROLL_SPECIES
    for (int k = 0; k < ns; k++) {
        double c[6];
        species_poly(P, k, T, c);
        dcv += ys[k] * poly_dcv(c, T);
        ysb[k] = cpb * (poly_cv(c, T) + kRuniv * P.inv_mw[k]);
    }
    *Tb += cpb * dcv;
    fill_y_vjp<NSMAX>(ns, U[0], U + 2 + DIM, ysb, Ub, Ub + 2 + DIM);
}

// reverse of transport(): adjoints of mu, k, D into the face state and the face temperature
template <int DIM, int NSMAX>
ABL_HD void transport_vjp(const Phys& P, int ns, const double* U, double T, double mub, double kb, double Db, double* Ub, double* Tb) {
    switch (P.transport) {
        case ABL_TRANSPORT_SUTHERLAND: {
            const double pr = 0.707, sc = 0.707, so = 111.0;
            const double m = sutherland_mu(T);
            const double cp = cp_at<DIM, NSMAX>(P, ns, U, T);
            const double mb = mub + kb * cp / pr + Db / (U[0] * sc);
            Ub[0] -= Db * m / (U[0] * U[0] * sc);
            *Tb += mb * m * (1.5 / T - 1.0 / (T + so));
            cp_at_vjp<DIM, NSMAX>(P, ns, U, T, kb * m / pr, Ub, Tb);
            return;
        }
        case ABL_TRANSPORT_CONSTANT_LEWIS: {
            const double cp = cp_at<DIM, NSMAX>(P, ns, U, T);
            const double k = P.mu * cp / P.k;
            const double D = k / (U[0] * cp * P.diff);
            const double kbt = kb + Db / (U[0] * cp * P.diff);
            Ub[0] -= Db * D / U[0];
            cp_at_vjp<DIM, NSMAX>(P, ns, U, T, kbt * P.mu / P.k - Db * D / cp, Ub, Tb);
            return;
        }
        default:
            return;  // constant properties
    }
}

// reverse of cell_aux(): aux = (T, u, Y) of a cell from its conserved state
template <int DIM, int NS>
__device__ __forceinline__ void cell_aux_vjp(const Phys& P, const double* u, const double* __restrict__ tmp, int c, const double* ab, double* Ub) {
    using D = Dims<DIM, NS>;
    const double irho = rcp64(u[0]);
    double irhob = 0;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        Ub[2 + d] += ab[1 + d] * irho;
        irhob += ab[1 + d] * u[2 + d];
    }
ABL_UNROLL_SPECIES
    for (int s = 0; s < NS; s++) {
        Ub[D::NE + s] += ab[1 + DIM + s] * irho;
        irhob += ab[1 + DIM + s] * u[D::NE + s];
    }
    Ub[0] -= irhob * irho * irho;
    if (ab[0] == 0.0) return;
    if (NS > 0 && P.eos == ABL_EOS_NASA7) {
        constexpr int NY = NS > 0 ? NS : 1;
        double ys[NY], ysb[NY];
        fill_y(NS, u[0], u + D::NE, ys);
        bool ok = true;
        const double T = temperature<DIM, NS>(P, NS, u, __ldg(tmp + c), &ok);
ABL_UNROLL_SPECIES
        for (int k = 0; k < NS; k++) ysb[k] = 0.0;
        nasa_temperature_vjp<DIM, NS>(P, NS, u, ys, T, ab[0], ysb, Ub);
        fill_y_vjp<NS>(NS, u[0], u + D::NE, ysb, Ub, Ub + D::NE);
    } else {
        internal_energy_vjp<DIM>(u, ab[0] * P.icv, Ub);
    }
}

// ---------------------------------------------------------------------------------------------------
// flux calculators: g[0..7] += d(mf, p12)/d(uL, aL, rhoL, pL, uR, aR, rhoR, pR)^T (mfb, p12b)
// ---------------------------------------------------------------------------------------------------
ABL_HD double sgn1(double m) { return m < 0 ? -1.0 : 1.0; }  // the derivative of dabs()

ABL_HD void ausm_vjp(const double* x, double mfb, double p12b, double* g) {
    const double uL = x[0], aL = x[1], rhoL = x[2], pL = x[3], uR = x[4], aR = x[5], rhoR = x[6], pR = x[7];
    const double iaR = rcp64(aR), iaL = rcp64(aL);
    const double Mm = uR * iaR, Mp = uL * iaL;
    const bool inM = fabs(Mm) <= 1.0, inP = fabs(Mp) <= 1.0;
    double sMm, sPm, sMp, sPp;
    if (inM) {
        sMm = -0.25 * sqr(Mm - 1.0);
        sPm = -sMm * (2.0 + Mm);
    } else {
        sMm = 0.5 * (Mm - fabs(Mm));
        sPm = sMm / Mm;
    }
    if (inP) {
        sMp = 0.25 * sqr(Mp + 1.0);
        sPp = sMp * (2.0 - Mp);
    } else {
        sMp = 0.5 * (Mp + fabs(Mp));
        sPp = sMp / Mp;
    }
    const double m = sMm + sMp;
    const double sPmb = p12b * pR, sPpb = p12b * pL;
    g[7] += p12b * sPm;
    g[3] += p12b * sPp;
    double mb;
    if (m < 0) {
        mb = mfb * aR * rhoR;
        g[5] += mfb * m * rhoR;
        g[6] += mfb * m * aR;
    } else {
        mb = mfb * aL * rhoL;
        g[1] += mfb * m * rhoL;
        g[2] += mfb * m * aL;
    }
    double sMmb = mb, sMpb = mb, Mmb = 0, Mpb = 0;
    if (inM) {
        sMmb -= sPmb * (2.0 + Mm);
        Mmb -= sPmb * sMm;
        Mmb -= sMmb * 0.5 * (Mm - 1.0);
    } else {
        sMmb += sPmb / Mm;
        Mmb -= sPmb * sPm / Mm;
        Mmb += sMmb * 0.5 * (1.0 - sgn1(Mm));
    }
    if (inP) {
        sMpb += sPpb * (2.0 - Mp);
        Mpb -= sPpb * sMp;
        Mpb += sMpb * 0.5 * (Mp + 1.0);
    } else {
        sMpb += sPpb / Mp;
        Mpb -= sPpb * sPp / Mp;
        Mpb += sMpb * 0.5 * (1.0 + sgn1(Mp));
    }
    g[4] += Mmb * iaR;
    g[5] -= Mmb * Mm * iaR;
    g[0] += Mpb * iaL;
    g[1] -= Mpb * Mp * iaL;
}

// derivatives of the AUSM+up splitting polynomials (Ausmpup in fv_physics.cuh)
struct AusmpupD {
    static ABL_HD double M2P(double m) { return 0.25 * sqr(m + 1.0); }
    static ABL_HD double M2M(double m) { return -0.25 * sqr(m - 1.0); }
    static ABL_HD double dM2P(double m) { return 0.5 * (m + 1.0); }
    static ABL_HD double dM2M(double m) { return -0.5 * (m - 1.0); }
    static ABL_HD double dM4P(double m) {
        if (fabs(m) >= 1.0) return 0.5 * (1.0 + sgn1(m));
        return dM2P(m) * (1.0 - 2.0 * M2M(m)) - 2.0 * M2P(m) * dM2M(m);
    }
    static ABL_HD double dM4M(double m) {
        if (fabs(m) >= 1.0) return 0.5 * (1.0 - sgn1(m));
        return dM2M(m) * (1.0 + 2.0 * M2P(m)) + 2.0 * M2M(m) * dM2P(m);
    }
    // d/dm and d/dfa of P5P, P5M
    static ABL_HD void dP5P(double m, double fa, double* dm, double* dfa) {
        if (fabs(m) >= 1.0) {
            const double e = m + 1E-30, m1 = 0.5 * (m + fabs(m));
            *dm = (0.5 * (1.0 + sgn1(m)) * e - m1) / (e * e);
            *dfa = 0.0;
            return;
        }
        const double al = 3.0 / 16.0 * (-4.0 + 5.0 * fa * fa);
        const double B = (2.0 - m) - 16.0 * al * m * M2M(m);
        *dm = dM2P(m) * B + M2P(m) * (-1.0 - 16.0 * al * (M2M(m) + m * dM2M(m)));
        *dfa = -30.0 * fa * m * M2P(m) * M2M(m);
    }
    static ABL_HD void dP5M(double m, double fa, double* dm, double* dfa) {
        if (fabs(m) >= 1.0) {
            const double e = m + 1E-30, m1 = 0.5 * (m - fabs(m));
            *dm = (0.5 * (1.0 - sgn1(m)) * e - m1) / (e * e);
            *dfa = 0.0;
            return;
        }
        const double al = 3.0 / 16.0 * (-4.0 + 5.0 * fa * fa);
        const double B = (-2.0 - m) + 16.0 * al * m * M2P(m);
        *dm = dM2M(m) * B + M2M(m) * (-1.0 + 16.0 * al * (M2P(m) + m * dM2P(m)));
        *dfa = 30.0 * fa * m * M2M(m) * M2P(m);
    }
};

ABL_HD void ausmpup_vjp(double mInf, double alpha, double ialpha, const double* x, double mfb, double p12b, double* g) {
    using A = Ausmpup<double>;
    using B = AusmpupD;
    const double uL = x[0], aL = x[1], rhoL = x[2], pL = x[3], uR = x[4], aR = x[5], rhoR = x[6], pR = x[7];
    const double Kp = 0.25, Ku = 0.75, sigma = 0.25;
    // forward
    const double rho12 = 0.5 * (rhoL + rhoR);
    const double a12 = 0.5 * (aL + aR) * ialpha;
    const double ia12 = rcp64(a12);
    const double mL = uL * ia12, mR = uR * ia12;
    const double mBar2 = (sqr(uL) + sqr(uR)) * (0.5 * ia12 * ia12);
    double fa = 1.0, mO = 0.0, xmax = 0.0;
    const double mInf2 = sqr(mInf);
    if (mInf > 0) {
        xmax = pmax(mBar2, mInf2);
        mO = sqrt(pmin(1.0, xmax));
        fa = mO * (2.0 - mO);
    }
    const double a2 = alpha * alpha;
    const double c = Kp * rcp64(fa);
    const double w1 = 1.0 - sigma * mBar2;
    const double w = pmax(w1, 0.0);
    const double dp = pR - pL;
    const double den = rho12 * a12 * a12 * a2;
    const double idn = rcp64(den);
    const double m12 = A::M4P(mL) + A::M4M(mR) - c * w * dp * idn;
    const double p5P = A::P5P(mL, fa), p5M = A::P5M(mR, fa);
    // reverse
    double mLb = 0, mRb = 0, fab = 0, a12b = 0, rho12b = 0, mBar2b = 0;
    const double vb = p12b * sqr(ialpha);
    g[3] += vb * p5P;
    g[7] += vb * p5M;
    const double K = Ku * rho12 * fa * a12 * a12 * a2 * (mR - mL);
    const double p5Pb = vb * (pL - p5M * K), p5Mb = vb * (pR - p5P * K);
    const double Q = -vb * Ku * p5P * p5M * a2;
    rho12b += Q * fa * a12 * a12 * (mR - mL);
    fab += Q * rho12 * a12 * a12 * (mR - mL);
    a12b += Q * rho12 * fa * 2.0 * a12 * (mR - mL);
    mRb += Q * rho12 * fa * a12 * a12;
    mLb -= Q * rho12 * fa * a12 * a12;
    double dm, dfa;
    B::dP5P(mL, fa, &dm, &dfa);
    mLb += p5Pb * dm;
    fab += p5Pb * dfa;
    B::dP5M(mR, fa, &dm, &dfa);
    mRb += p5Mb * dm;
    fab += p5Mb * dfa;
    double m12b;
    if (m12 > 0) {
        m12b = mfb * a12 * rhoL;
        a12b += mfb * m12 * rhoL;
        g[2] += mfb * a12 * m12;
    } else {
        m12b = mfb * a12 * rhoR;
        a12b += mfb * m12 * rhoR;
        g[6] += mfb * a12 * m12;
    }
    mLb += m12b * B::dM4P(mL);
    mRb += m12b * B::dM4M(mR);
    const double tb = -m12b;
    const double cb = tb * w * dp * idn, wb = tb * c * dp * idn, dpb = tb * c * w * idn, idnb = tb * c * w * dp;
    const double denb = -idnb * idn * idn;
    fab -= cb * Kp / (fa * fa);
    if (!(w1 < 0.0)) mBar2b -= sigma * wb;
    g[7] += dpb;
    g[3] -= dpb;
    rho12b += denb * a12 * a12 * a2;
    a12b += denb * rho12 * 2.0 * a12 * a2;
    if (mInf > 0) {
        const double mOb = fab * (2.0 - 2.0 * mO);
        const double mO2b = mO > 0 ? mOb / (2.0 * mO) : 0.0;
        if (!(1.0 < xmax) && !(mBar2 < mInf2)) mBar2b += mO2b;
    }
    double ia12b = mBar2b * (sqr(uL) + sqr(uR)) * ia12;
    g[0] += mBar2b * uL * ia12 * ia12 + mLb * ia12;
    g[4] += mBar2b * uR * ia12 * ia12 + mRb * ia12;
    ia12b += mLb * uL + mRb * uR;
    a12b -= ia12b * ia12 * ia12;
    g[1] += 0.5 * a12b * ialpha;
    g[5] += 0.5 * a12b * ialpha;
    g[2] += 0.5 * rho12b;
    g[6] += 0.5 * rho12b;
}

// any calculator: eight tangent evaluations (exact Riemann, average)
ABL_HD void calc_vjp_tangents(const Phys& P, const double* x, double mfb, double p12b, double* g, bool* rok) {
#pragma unroll 1
    for (int i = 0; i < 8; i++) {
        Dual xi[8];
#pragma unroll
        for (int j = 0; j < 8; j++) xi[j] = Dual(x[j], i == j ? 1.0 : 0.0);
        Dual mf, p12;
        flux_calc<Dual>(P, xi[0], xi[1], xi[2], xi[3], xi[4], xi[5], xi[6], xi[7], &mf, &p12, rok);
        g[i] += mfb * mf.d + p12b * p12.d;
    }
}

template <int FK>
ABL_HD void calc_vjp(const Phys& P, const double* x, double mfb, double p12b, double* g, bool* rok) {
    const int kind = FK >= 0 ? FK : P.flux;
    if (kind == ABL_FLUX_AUSM)
        ausm_vjp(x, mfb, p12b, g);
    else if (kind == ABL_FLUX_AUSMPUP)
        ausmpup_vjp(P.minf, P.alpha, P.ialpha, x, mfb, p12b, g);
    else
        calc_vjp_tangents(P, x, mfb, p12b, g, rok);
}

// ---------------------------------------------------------------------------------------------------
// face fluxes backwards
// ---------------------------------------------------------------------------------------------------
// One side of the advection flux backwards: eb, pb, irhob, velb and ub arrive with the upwind terms; the
// flux calculator's adjoints of (u.n, a, rho, p) on this side are g[0..3]. ub is this side's face state.
template <int DIM, int NS>
__device__ __forceinline__ void advection_side_vjp(const Phys& P, const double* norm, const double* u, double irho, const Decoded<double>& dd,
                                                   const double* g, double eb, double pb, double irhob, double* velb, double* ub) {
    ub[0] += g[2];
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        velb[d] += g[0] * norm[d];
        ub[2 + d] += velb[d] * irho;
        irhob += velb[d] * u[2 + d];
    }
    ub[0] -= irhob * irho * irho;
    decode_vjp<DIM, NS>(P, NS, u, dd, eb, g[1], pb + g[3], ub);
}

// advection (NavierStokesTransport::AdvectionFlux + SpeciesTransport::AdvectionFlux) backwards: fb = flux
// adjoint, ubL and ubR = adjoints of the two projected face states
template <int DIM, int NS, int FK>
__device__ __forceinline__ void advection_vjp(const Phys& P, const double* normal, double areaMag, const double* uL, const double* uR, double gsL, double gsR,
                                              bool adv, bool spadv, const double* fb, double* ubL, double* ubR, bool* ok, bool* rok) {
    using D = Dims<DIM, NS>;
    const double iA = rcp64(areaMag);
    double norm[DIM];
#pragma unroll
    for (int d = 0; d < DIM; d++) norm[d] = normal[d] * iA;
    const auto dL = decode<DIM, NS>(P, NS, uL, gsL, ok);
    const auto dR = decode<DIM, NS>(P, NS, uR, gsR, ok);
    const double irL = rcp64(uL[0]), irR = rcp64(uR[0]);
    double velL[DIM], velR[DIM], unL = 0, unR = 0;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        velL[d] = uL[2 + d] * irL;
        unL += velL[d] * norm[d];
        velR[d] = uR[2 + d] * irR;
        unR += velR[d] * norm[d];
    }
    const double x[8] = {unL, dL.a, uL[0], dL.p, unR, dR.a, uR[0], dR.p};
    double mf, p12;
    const int dir = flux_calc_k<FK, double>(P, x[0], x[1], x[2], x[3], x[4], x[5], x[6], x[7], &mf, &p12, rok);
    const double mA = mf * areaMag;
    // LEFT upwinds side L, RIGHT side R, no direction half of each; for the species anything but LEFT is R
    const double wL = dir == ABL_DIR_LEFT ? 1.0 : (dir == ABL_DIR_RIGHT ? 0.0 : 0.5), wR = 1.0 - wL;
    double mfb = 0, p12b = 0, ebL = 0, ebR = 0, pbL = 0, pbR = 0, ibL = 0, ibR = 0, vbL[DIM], vbR[DIM];
#pragma unroll
    for (int d = 0; d < DIM; d++) vbL[d] = vbR[d] = 0.0;
ABL_UNROLL_SPECIES
    for (int k = 0; k < D::NC; k++) ubL[k] = ubR[k] = 0.0;
    if (adv) {
        double v2L = 0, v2R = 0;
#pragma unroll
        for (int d = 0; d < DIM; d++) {
            v2L += velL[d] * velL[d];
            v2R += velR[d] * velR[d];
        }
        const double HL = dL.e + 0.5 * v2L + dL.p * irL, HR = dR.e + 0.5 * v2R + dR.p * irR;
        mfb = areaMag * fb[0];
        double sacc = (wL * HL + wR * HR) * fb[1];
#pragma unroll
        for (int n = 0; n < DIM; n++) {
            p12b += normal[n] * fb[2 + n];
            sacc += (wL * velL[n] + wR * velR[n]) * fb[2 + n];
        }
        mfb += areaMag * sacc;
        const double Hb = mA * fb[1];
        ebL = wL * Hb;
        ebR = wR * Hb;
        pbL = ebL * irL;
        pbR = ebR * irR;
        ibL = ebL * dL.p;
        ibR = ebR * dR.p;
#pragma unroll
        for (int n = 0; n < DIM; n++) {
            vbL[n] = ebL * velL[n] + wL * mA * fb[2 + n];
            vbR[n] = ebR * velR[n] + wR * mA * fb[2 + n];
        }
    }
    if (NS > 0 && spadv && dir == ABL_DIR_NA && P.sp_compact) {
        // compact process, no direction: flux_s = mA (rhoY_L + rhoY_R) / (rho_L + rho_R) (both halves)
        const double irm = 1.0 / (0.5 * (uL[0] + uR[0]));
ABL_UNROLL_SPECIES
        for (int s = 0; s < NS; s++) {
            const double num = 0.5 * (uL[D::NE + s] + uR[D::NE + s]);
            mfb += areaMag * num * irm * fb[D::NE + s];
            const double yb = 0.5 * mA * irm * fb[D::NE + s], rb = yb * num * irm;
            ubL[D::NE + s] = yb;
            ubR[D::NE + s] = yb;
            ubL[0] -= rb;
            ubR[0] -= rb;
        }
    } else if (NS > 0 && spadv) {
        const bool left = dir == ABL_DIR_LEFT;
        const double ir = left ? irL : irR;
        double ib = 0;
ABL_UNROLL_SPECIES
        for (int s = 0; s < NS; s++) {
            const double ry = left ? uL[D::NE + s] : uR[D::NE + s], Yb = mA * fb[D::NE + s];
            mfb += areaMag * (ry * ir) * fb[D::NE + s];
            ubL[D::NE + s] = left ? Yb * ir : 0.0;
            ubR[D::NE + s] = left ? 0.0 : Yb * ir;
            ib += Yb * ry;
        }
        if (left)
            ibL += ib;
        else
            ibR += ib;
    }
    double g[8] = {0, 0, 0, 0, 0, 0, 0, 0};
    if (mfb != 0.0 || p12b != 0.0) calc_vjp<FK>(P, x, mfb, p12b, g, rok);
    advection_side_vjp<DIM, NS>(P, norm, uL, irL, dL, g, ebL, pbL, ibL, vbL, ubL);
    advection_side_vjp<DIM, NS>(P, norm, uR, irR, dR, g + 4, ebR, pbR, ibR, vbR, ubR);
}

// diffusion (NavierStokesTransport::DiffusionFlux, SpeciesTransport diffusion) backwards. fs, fa and gf are
// the face state, aux and aux gradient (averages of the two cells); each side receives half of the adjoints
// fsb (state), fab (T, u) and of the aux gradient's, which is made of one number per aux component and the
// area normal n (aux_gradient_adjoint). gf and the gradient's adjoint hold the velocity part in the symmetric
// form of GradComps; the adjoint of du_c/dx_d is that of du_d/dx_c:
//   T: -gs n,   u_c, d: -(gs_c n_d + gs_d n_c - 2/3 delta_cd gs.n),   Y_s: -gs n
template <int DIM, int NS>
__device__ __forceinline__ void diffusion_vjp(const Phys& P, const double* normal, const double* fs, const double* fa, const double* gf, bool dif,
                                              bool spdif, const double* fb, double* fsb, double* fab, double* gs) {
    using D = Dims<DIM, NS>;
    using GC = GradComps<DIM, NS>;
ABL_UNROLL_SPECIES
    for (int k = 0; k < D::NC; k++) fsb[k] = 0.0;
ABL_UNROLL_SPECIES
    for (int k = 0; k < D::NA; k++) gs[k] = 0.0;
#pragma unroll
    for (int k = 0; k < 1 + DIM; k++) fab[k] = 0.0;
    double mu, kc, diff;
    transport<DIM, NS>(P, NS, fs, fa[0], &mu, &kc, &diff);
    double mub = 0, kb = 0, Db = 0;
    if (dif) {
        double divVel = 0;
#pragma unroll
        for (int c = 0; c < DIM; ++c) divVel += gf[GC::sym(c, c)];
#pragma unroll
        for (int c = 0; c < DIM; ++c) {
            double sn = 0;  // row c of the stress over mu, times n
#pragma unroll
            for (int d = 0; d < DIM; ++d)
                sn += ((d == c) ? 2.0 * (gf[GC::sym(c, c)] - divVel / 3.0) : gf[GC::sym(c, d)]) * normal[d];
            const double w = fb[2 + c] + fa[1 + c] * fb[1];
            fab[1 + c] = -mu * sn * fb[1];
            mub -= w * sn;
            gs[1 + c] = mu * w;
            kb -= normal[c] * gf[c] * fb[1];
        }
        gs[0] = kc * fb[1];
    }
    if constexpr (NS > 0) {
        if (spdif) {
            const double density = fs[0];
            double rhob = 0, Tb = 0;
ABL_UNROLL_SPECIES
            for (int s = 0; s < NS; ++s) {
                double hs = 0.0, cps = 0.0;
                if (P.eos == ABL_EOS_NASA7) {
                    double c[6];
                    species_poly(P, s, fa[0], c);
                    const double r = kRuniv * P.inv_mw[s];
                    hs = poly_e(c, fa[0]) + r * fa[0];
                    cps = poly_cv(c, fa[0]) + r;
                }
                // one constant D_k per species (no state dependence), or the transport model's D
                const double Ds = P.diff_k ? P.diff_k[s] : diff;
                double gn = 0;
#pragma unroll
                for (int d = 0; d < DIM; ++d) gn += normal[d] * gf[GC::Y + s * DIM + d];
                const double q = fb[D::NE + s] + hs * fb[1];
                rhob -= q * Ds * gn;
                if (!P.diff_k) Db -= q * density * gn;
                gs[1 + DIM + s] = q * density * Ds;
                Tb -= density * Ds * gn * fb[1] * cps;
            }
            fsb[0] += rhob;
            fab[0] += Tb;
        }
    }
    transport_vjp<DIM, NS>(P, NS, fs, fa[0], mub, kb, Db, fsb, &fab[0]);
}

// ga += half of the aux gradient's adjoint of a face with area normal n (see diffusion_vjp)
template <int DIM, int NS>
__device__ __forceinline__ void aux_gradient_adjoint(const double* n, const double* gs, double* ga) {
    using GC = GradComps<DIM, NS>;
    double tr = 0;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        ga[d] -= 0.5 * gs[0] * n[d];
        tr += gs[1 + d] * n[d];
    }
#pragma unroll
    for (int c = 0; c < DIM; c++)
#pragma unroll
        for (int d = c; d < DIM; d++) ga[GC::sym(c, d)] -= 0.5 * (gs[1 + c] * n[d] + gs[1 + d] * n[c] - (c == d ? 2.0 / 3.0 * tr : 0.0));
ABL_UNROLL_SPECIES
    for (int s = 0; s < NS; s++)
#pragma unroll
        for (int d = 0; d < DIM; d++) ga[GC::Y + s * DIM + d] -= 0.5 * gs[1 + DIM + s] * n[d];
}
// ab += sign times the weights w contracted with the aux gradient's adjoint ga (the reverse of
// sum_d w_d (a_n - a_c) for T, u and Y)
template <int DIM, int NS>
__device__ __forceinline__ void contract_aux(double sign, const double* w, const double* ga, double* ab) {
    using GC = GradComps<DIM, NS>;
#pragma unroll
    for (int d = 0; d < DIM; d++) {
        const double x = sign * w[d];
        ab[0] += x * ga[d];
#pragma unroll
        for (int c = 0; c < DIM; c++) ab[1 + c] += x * ga[GC::sym(c, d)];
ABL_UNROLL_SPECIES
        for (int s = 0; s < NS; s++) ab[1 + DIM + s] += x * ga[GC::Y + s * DIM + d];
    }
}

// ---------------------------------------------------------------------------------------------------
// the adjoint row of a non-owned cell's side of one face: [state NC][limited gradient NC*DIM][aux NA][aux gradient GradComps::A]
template <int DIM, int NS>
struct AdjRow {
    using D = Dims<DIM, NS>;
    static constexpr int U = 0, G = D::NC, A = D::NC + D::NC * DIM, GA = D::NC + D::NC * DIM + D::NA;
    static constexpr int N = GA + GradComps<DIM, NS>::A;
    // shared-memory record of one face, [comp][face of the tile]: the diffusion pass leaves gs (NA), fab
    // (1+DIM) and fsb's density and species (1+NS; its others are 0), the advection pass ubL and ubR
    static constexpr int FG = 0, FA = D::NA, FS = D::NA + 1 + DIM;
    static constexpr int R = 2 * D::NC;
    static_assert(FS + 1 + NS <= R, "the advection pass's record is the larger");
};

// dF_L/dflux = -1/V_L, dF_R/dflux = +1/V_R on owned cells: the flux adjoint of a face
template <int DIM, int NS>
__device__ __forceinline__ void flux_adjoint(const DevMesh& M, int2 lr, const double* __restrict__ Fb, double* fb) {
    using D = Dims<DIM, NS>;
    const double iL = M.kind[lr.x] == ABL_CELL_OWNED ? -M.ivol[lr.x] : 0.0;
    const double iR = M.kind[lr.y] == ABL_CELL_OWNED ? M.ivol[lr.y] : 0.0;
ABL_UNROLL_SPECIES
    for (int k = 0; k < D::NC; k++) {
        // a non-owned row of Fbar is not read: it may hold anything
        const double l = iL != 0.0 ? __ldg(Fb + (size_t)lr.x * D::NC + k) * iL : 0.0;
        const double r = iR != 0.0 ? __ldg(Fb + (size_t)lr.y * D::NC + k) * iR : 0.0;
        fb[k] = l + r;
    }
}

// the record of the face's non-owned side in nbrec, or null: *side is that side
template <int DIM, int NS>
__device__ __forceinline__ double* nonowned_row(const DevMesh& M, int i, int2 lr, double* nbrec, int* side) {
    const int nb = M.tf_nb[i];
    if (nb < 0) return nullptr;
    *side = M.kind[lr.x] != ABL_CELL_OWNED ? 0 : 1;
    return nbrec + (size_t)nb * AdjRow<DIM, NS>::N;
}

// ---------------------------------------------------------------------------------------------------
// cell step: limiter and least-squares gradient backwards (the limiter recomputed), aux-gradient self
// term; writes the per-cell records the gather reads
template <int DIM, int NS>
struct AdjOut {  // component by component, as the gradients: [comp][cell]
    double* gb;     // adjoint of the unlimited state gradient
    double* beta;   // limiter term for the minimising neighbour
    int* fstar;     // face of that neighbour, -1 for none
    double* gab;    // adjoint of the aux gradient
    double* ub;     // state adjoint, own terms
    double* ab;     // aux adjoint, own terms
};

// forward records of k_gradient<..., REC = true>: unlimited gradient, applied limiter factor, and the
// cone entry of the minimising face per component
struct GradRec {
    const double* graw;
    const double* phi;
    const int* ist;
};

// the state's part: ub and gt are the adjoints of the cell's state and limited gradient from its faces
template <int DIM, int NS, int LIM>
__device__ __forceinline__ void cell_vjp_state(const DevMesh& M, const Phys& P, int c, const double* __restrict__ U, double* ub, const double* gt,
                                               const GradRec& rec, const AdjOut<DIM, NS>& out, bool do_state) {
    using D = Dims<DIM, NS>;
    using GC = GradComps<DIM, NS>;
    const uint8_t kind = M.kind[c];
    const bool state = do_state && (kind == ABL_CELL_OWNED || kind == ABL_CELL_HALO);
    double gbar[D::NC * DIM];
ABL_UNROLL_SPECIES
    for (int k = 0; k < D::NC; k++) {
        double beta = 0.0;
        int fst = -1;
#pragma unroll
        for (int d = 0; d < DIM; d++) gbar[k * DIM + d] = 0.0;
        if (state) {
            // g~ = phi g (0 when cancelled): g-bar = phi g~-bar, plus the limiter's own dependence on g and on
            // the minimising neighbour through r = (u_n - u_c) / (2 g . dx)
            double g[DIM];
#pragma unroll
            for (int d = 0; d < DIM; d++) g[d] = __ldg(rec.graw + (k * DIM + d) * M.gs + c);
            const double ph = __ldg(rec.phi + k * M.gs + c);
            const int i = __ldg(rec.ist + k * M.gs + c);
            double phib = 0;
#pragma unroll
            for (int d = 0; d < DIM; d++) {
                gbar[k * DIM + d] = ph * gt[k * DIM + d];
                phib += gt[k * DIM + d] * g[d];
            }
            if (i >= 0 && phib != 0.0) {
                const int2 ce = M.cone[i];
                const int f = ce.x, n = ce.y & kConeNbr, sc = (ce.y & kConeSide) ? 1 : 0;
                double v[DIM], denom = 0;
#pragma unroll
                for (int d = 0; d < DIM; d++) {
                    v[d] = __ldg(M.fdx + 6 * (size_t)f + 3 * sc + d) - __ldg(M.fdx + 6 * (size_t)f + 3 * (1 - sc) + d);
                    denom += g[d] * v[d];
                }
                const double idn = rcp64(denom);
                const double r = 0.5 * (__ldg(U + (size_t)n * D::NC + k) - __ldg(U + (size_t)c * D::NC + k)) * idn;
                const double dl = limiter_k<LIM, Dual>(P.limiter, Dual(r, 1.0)).d;
                const double rb = dl * phib;
                if (rb != 0.0 && isfinite(rb) && isfinite(r)) {
                    beta = 0.5 * rb * idn;  // d r / d (u_n - u_c) = 1 / (2 denom)
                    fst = f;
                    ub[k] -= beta;
#pragma unroll
                    for (int d = 0; d < DIM; d++) gbar[k * DIM + d] -= r * rb * idn * v[d];  // d r / d denom = -r / denom
                }
            }
        }
        out.beta[k * M.gs + c] = beta;
        out.fstar[k * M.gs + c] = fst;
    }
    if (state) {
        // g = sum_f w_f (u_n - u_c): the own-cell term, with the cell's summed weights
#pragma unroll
        for (int d = 0; d < DIM; d++) {
            const double ws = __ldg(M.wsum + 6 * (size_t)c + d);
ABL_UNROLL_SPECIES
            for (int k = 0; k < D::NC; k++) ub[k] -= ws * gbar[k * DIM + d];
        }
    }
    if (out.gb) store_comps<GC::S>(out.gb, M.gs, c, gbar);
    store_comps<D::NC>(out.ub, M.gs, c, ub);
}

// the aux fields' part: ab and ga are the adjoints of the cell's aux and aux gradient from its faces
template <int DIM, int NS>
__device__ __forceinline__ void cell_vjp_aux(const DevMesh& M, int c, double* ab, const double* ga, const AdjOut<DIM, NS>& out, bool do_aux) {
    using D = Dims<DIM, NS>;
    using GC = GradComps<DIM, NS>;
    const bool auxg = do_aux && M.kind[c] != ABL_CELL_HALO_OUTER;
    if (auxg) {
        double ws[DIM];
#pragma unroll
        for (int d = 0; d < DIM; d++) ws[d] = __ldg(M.wsum + 6 * (size_t)c + 3 + d);
        contract_aux<DIM, NS>(-1.0, ws, ga, ab);
    }
    if (out.gab) {
ABL_UNROLL_SPECIES
        for (int k = 0; k < GC::A; k++) out.gab[k * M.gs + c] = auxg ? ga[k] : 0.0;
    }
    store_comps<D::NA>(out.ab, M.gs, c, ab);
}

// ---------------------------------------------------------------------------------------------------
// kernels
// ---------------------------------------------------------------------------------------------------
// most threads of a CTA, and the resident CTAs per SM that the register budget targets: 128 registers without
// species, 168 with up to 5, 255 with more
template <int NS>
struct AdjBlocks {
    static constexpr int threads = NS == 0 ? 256 : 128;
    static constexpr int tile = NS == 0 ? 2 : (NS > 5 ? 2 : 3);
};

// One CTA per tile, one thread per face and then one per cell, as the forward pass: the faces' adjoints
// go to one shared-memory record per face, and every cell sums its faces' records in ascending face order
// in registers (no atomics, no ordering between the faces). The diffusion and the advection flux take one
// such round each: a round's record is a third of both, and so are the live registers. Bound by the latency
// of its loads and FP64 chains. Two lanes per face, both evaluating what couples the sides, with per-cell
// accumulators in shared memory that the faces updated colour by colour, took 114 M warp instructions at
// 64^3 cells; this takes 60 M (523 -> 213 us).
template <int DIM, int NS, int FK, int LIM>
__global__ void __launch_bounds__(AdjBlocks<NS>::threads, AdjBlocks<NS>::tile) k_tile_adjoint(DevMesh M, Phys P, const double* __restrict__ U, const double* __restrict__ tmp,
                                                                          const double* __restrict__ grad, const double* __restrict__ agrad,
                                                                          const double* __restrict__ Fb, GradRec rec, AdjOut<DIM, NS> out,
                                                                          double* __restrict__ nbrec, int do_state, int do_aux, int* status) {
    using D = Dims<DIM, NS>;
    using GC = GradComps<DIM, NS>;
    using AR = AdjRow<DIM, NS>;
    extern __shared__ double srec[];  // [AR::R][tile faces]
    const int t = blockIdx.x;
    const int cb = M.tile_cell_ptr[t], ce = M.tile_cell_ptr[t + 1];
    const int fb = M.tile_face_ptr[t], fe = M.tile_face_ptr[t + 1], nf = fe - fb;
    bool ok = true, rok = true;
    const bool dif = P.diffusion && P.transport != ABL_TRANSPORT_NONE;
    const bool spdif = NS > 0 && P.sp_dif && P.transport != ABL_TRANSPORT_NONE;
    const bool adv = P.advection && P.flux != ABL_FLUX_OFF;
    const bool spadv = NS > 0 && P.sp_adv && P.flux != ABL_FLUX_OFF;
    const bool lsq = P.recon == ABL_RECON_LEASTSQUARES;
    if (dif || spdif) {
        for (int i = fb + threadIdx.x; i < fe; i += blockDim.x) {
            const int2 lr = M.tf_cells[i];
            double normal[DIM], fdx[7], flb[D::NC], fs[D::NC], fa[D::NA], gf[GC::A];
            face_geometry<DIM, double>(M, i, normal, fdx);
            flux_adjoint<DIM, NS>(M, lr, Fb, flb);
            double wl = 0, wr = 0;
            {
                double cL[D::NC], cR[D::NC], aL[D::NA], aR[D::NA];
                load_state<DIM, NS>(U, lr.x, cL);
                load_state<DIM, NS>(U, lr.y, cR);
                cell_aux<DIM, NS>(P, cL, tmp, lr.x, aL);
                cell_aux<DIM, NS>(P, cR, tmp, lr.y, aR);
ABL_UNROLL_SPECIES
                for (int k = 0; k < D::NC; k++) fs[k] = cL[k] * 0.5 + cR[k] * 0.5;
ABL_UNROLL_SPECIES
                for (int k = 0; k < D::NA; k++) fa[k] = aL[k] * 0.5 + aR[k] * 0.5;
                if constexpr (DIM == 1) {
                    // in 1D the face gradient is the two-cell LeastSquares stencil's
                    face_weights_1d(fdx, &wl, &wr);
ABL_UNROLL_SPECIES
                    for (int k = 0; k < D::NA; k++) gf[k] = aL[k] * wl + aR[k] * wr;
                }
            }
            if constexpr (DIM > 1) {
                double gL[GC::A], gR[GC::A];
                load_comps<GC::A>(agrad, M.gs, lr.x, gL);
                load_comps<GC::A>(agrad, M.gs, lr.y, gR);
ABL_UNROLL_SPECIES
                for (int k = 0; k < GC::A; k++) gf[k] = 0.5 * gL[k] + 0.5 * gR[k];
            }
            double fsb[D::NC], fab[1 + DIM], gs[D::NA];
            diffusion_vjp<DIM, NS>(P, normal, fs, fa, gf, dif, spdif, flb, fsb, fab, gs);
            double* r = srec + (i - fb);
ABL_UNROLL_SPECIES
            for (int k = 0; k < D::NA; k++) r[(AR::FG + k) * nf] = gs[k];
#pragma unroll
            for (int k = 0; k < 1 + DIM; k++) r[(AR::FA + k) * nf] = fab[k];
            r[AR::FS * nf] = fsb[0];
ABL_UNROLL_SPECIES
            for (int k = 0; k < NS; k++) r[(AR::FS + 1 + k) * nf] = fsb[D::NE + k];
            int side;
            if (double* nr = nonowned_row<DIM, NS>(M, i, lr, nbrec, &side)) {
                double ga[GC::A];
ABL_UNROLL_SPECIES
                for (int k = 0; k < GC::A; k++) ga[k] = 0.0;
                aux_gradient_adjoint<DIM, NS>(normal, gs, ga);
ABL_UNROLL_SPECIES
                for (int k = 0; k < D::NC; k++) nr[AR::U + k] = 0.5 * fsb[k];
ABL_UNROLL_SPECIES
                for (int k = 0; k < D::NA; k++)
                    nr[AR::A + k] = (k < 1 + DIM ? 0.5 * fab[k < 1 + DIM ? k : 0] : 0.0) + (DIM == 1 ? 2.0 * (side ? wr : wl) * ga[k] : 0.0);
ABL_UNROLL_SPECIES
                for (int k = 0; k < GC::A; k++) nr[AR::GA + k] = DIM == 1 ? 0.0 : ga[k];
            }
        }
        __syncthreads();
        for (int j = cb + threadIdx.x; j < ce; j += blockDim.x) {
            const int c = M.tile_cells[j];
            double ab[D::NA], ga[GC::A], ub[D::NC];
ABL_UNROLL_SPECIES
            for (int k = 0; k < D::NA; k++) ab[k] = 0.0;
ABL_UNROLL_SPECIES
            for (int k = 0; k < GC::A; k++) ga[k] = 0.0;
ABL_UNROLL_SPECIES
            for (int k = 0; k < D::NC; k++) ub[k] = 0.0;
            for (int e = M.tc_fptr[j]; e < M.tc_fptr[j + 1]; e++) {
                const uint16_t code = M.tc_face[e];
                const int q = code & 0x7fff;
                const double* r = srec + q;
                double normal[DIM], fdx[7], gs[D::NA];
                face_geometry<DIM, double>(M, fb + q, normal, fdx);
ABL_UNROLL_SPECIES
                for (int k = 0; k < D::NA; k++) gs[k] = r[(AR::FG + k) * nf];
                if constexpr (DIM == 1) {
                    double wl, wr;
                    face_weights_1d(fdx, &wl, &wr);
                    double g1[GC::A];  // (T, u, Y), as the aux components
ABL_UNROLL_SPECIES
                    for (int k = 0; k < GC::A; k++) g1[k] = 0.0;
                    aux_gradient_adjoint<DIM, NS>(normal, gs, g1);
ABL_UNROLL_SPECIES
                    for (int k = 0; k < D::NA; k++) ab[k] += 2.0 * ((code & 0x8000) ? wr : wl) * g1[k];
                } else {
                    aux_gradient_adjoint<DIM, NS>(normal, gs, ga);
                }
#pragma unroll
                for (int k = 0; k < 1 + DIM; k++) ab[k] += 0.5 * r[(AR::FA + k) * nf];
                ub[0] += 0.5 * r[AR::FS * nf];
ABL_UNROLL_SPECIES
                for (int k = 0; k < NS; k++) ub[D::NE + k] += 0.5 * r[(AR::FS + 1 + k) * nf];
            }
            cell_vjp_aux<DIM, NS>(M, c, ab, ga, out, do_aux);
            store_comps<D::NC>(out.ub, M.gs, c, ub);  // read back below, by the same thread
        }
        __syncthreads();
    }
    if (adv || spadv) {
        for (int i = fb + threadIdx.x; i < fe; i += blockDim.x) {
            const int2 lr = M.tf_cells[i];
            double normal[DIM], fdx[7], uL[D::NC], uR[D::NC], flb[D::NC];
            face_geometry<DIM, double>(M, i, normal, fdx);
            load_state<DIM, NS>(U, lr.x, uL);
            load_state<DIM, NS>(U, lr.y, uR);
            if (lsq) {
                double gL[GC::S], gR[GC::S];
                load_comps<GC::S>(grad, M.gs, lr.x, gL);
                load_comps<GC::S>(grad, M.gs, lr.y, gR);
ABL_UNROLL_SPECIES
                for (int k = 0; k < D::NC; k++) {
                    double dotL = 0, dotR = 0;
#pragma unroll
                    for (int d = 0; d < DIM; d++) {
                        dotL += gL[k * DIM + d] * fdx[d];
                        dotR += gR[k * DIM + d] * fdx[3 + d];
                    }
                    uL[k] += dotL;
                    uR[k] += dotR;
                }
            }
            double gsL = 300.0, gsR = 300.0;
            if (NS > 0 && P.eos == ABL_EOS_NASA7) {
                const double TL = __ldg(tmp + lr.x), TR = __ldg(tmp + lr.y);
                gsL = TL * .67 + .33 * TR;
                gsR = TL * .33 + .67 * TR;
            }
            flux_adjoint<DIM, NS>(M, lr, Fb, flb);
            double ubL[D::NC], ubR[D::NC];
            advection_vjp<DIM, NS, FK>(P, normal, fdx[6], uL, uR, gsL, gsR, adv, spadv, flb, ubL, ubR, &ok, &rok);
            double* r = srec + (i - fb);
ABL_UNROLL_SPECIES
            for (int k = 0; k < D::NC; k++) {
                r[k * nf] = ubL[k];
                r[(D::NC + k) * nf] = ubR[k];
            }
            int side;
            if (double* nr = nonowned_row<DIM, NS>(M, i, lr, nbrec, &side)) {
                const bool first = !(dif || spdif);
ABL_UNROLL_SPECIES
                for (int k = 0; k < D::NC; k++) {
                    const double v = side ? ubR[k] : ubL[k];
                    nr[AR::U + k] = first ? v : nr[AR::U + k] + v;
#pragma unroll
                    for (int d = 0; d < DIM; d++) nr[AR::G + k * DIM + d] = lsq ? v * fdx[side ? 3 + d : d] : 0.0;
                }
            }
        }
        __syncthreads();
    }
    for (int j = cb + threadIdx.x; j < ce; j += blockDim.x) {
        const int c = M.tile_cells[j];
        double ub[D::NC], gt[D::NC * DIM];
ABL_UNROLL_SPECIES
        for (int k = 0; k < D::NC; k++) ub[k] = (dif || spdif) ? out.ub[k * M.gs + c] : 0.0;
ABL_UNROLL_SPECIES
        for (int k = 0; k < D::NC * DIM; k++) gt[k] = 0.0;
        if (adv || spadv)
            for (int e = M.tc_fptr[j]; e < M.tc_fptr[j + 1]; e++) {
                const uint16_t code = M.tc_face[e];
                const int q = code & 0x7fff, side = code >> 15;
                const double* r = srec + side * D::NC * nf + q;
                const double* geo = M.tf_geo + 10 * geo_record(M, fb + q) + 3 + 3 * side;
                double dx[DIM];
#pragma unroll
                for (int d = 0; d < DIM; d++) dx[d] = lsq ? __ldg(geo + d) : 0.0;
                // u_face = u_cell + g . dx: the identity part to the state, the outer product with dx to the gradient
ABL_UNROLL_SPECIES
                for (int k = 0; k < D::NC; k++) {
                    const double v = r[k * nf];
                    ub[k] += v;
#pragma unroll
                    for (int d = 0; d < DIM; d++) gt[k * DIM + d] += v * dx[d];
                }
            }
        cell_vjp_state<DIM, NS, LIM>(M, P, c, U, ub, gt, rec, out, do_state);
        if (!(dif || spdif)) {
            double ab[D::NA], ga[GC::A];
ABL_UNROLL_SPECIES
            for (int k = 0; k < D::NA; k++) ab[k] = 0.0;
ABL_UNROLL_SPECIES
            for (int k = 0; k < GC::A; k++) ga[k] = 0.0;
            cell_vjp_aux<DIM, NS>(M, c, ab, ga, out, do_aux);
        }
    }
    if (!ok) atomicOr(status, kStatusEos);
    if (!rok) atomicOr(status, kStatusRiemann);
}

template <int DIM, int NS, int LIM>
__global__ void __launch_bounds__(128) k_adjoint_nonowned(DevMesh M, Phys P, const double* __restrict__ U, const double* __restrict__ nbrec,
                                                          GradRec rec, AdjOut<DIM, NS> out, int do_state, int do_aux) {
    using AR = AdjRow<DIM, NS>;
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= M.n_nonowned) return;
    const int c = M.nonowned[j];
    double acc[AR::N];
ABL_UNROLL_SPECIES
    for (int k = 0; k < AR::N; k++) acc[k] = 0.0;
    for (int i = M.cone_ptr[c]; i < M.cone_ptr[c + 1]; i++) {
        const int nb = M.face_nb[M.cone[i].x];
        if (nb < 0) continue;
        const double* r = nbrec + (size_t)nb * AR::N;
ABL_UNROLL_SPECIES
        for (int k = 0; k < AR::N; k++) acc[k] += r[k];
    }
    cell_vjp_aux<DIM, NS>(M, c, acc + AR::A, acc + AR::GA, out, do_aux);
    cell_vjp_state<DIM, NS, LIM>(M, P, c, U, acc + AR::U, acc + AR::G, rec, out, do_state);
}

template <int DIM, int NS>
__global__ void __launch_bounds__(128) k_adjoint_gather(DevMesh M, Phys P, const double* __restrict__ U, const double* __restrict__ tmp,
                                                        AdjOut<DIM, NS> in, double* __restrict__ Ub, int do_state, int do_aux, int* status) {
    using D = Dims<DIM, NS>;
    using GC = GradComps<DIM, NS>;
    const int m = blockIdx.x * blockDim.x + threadIdx.x;
    if (m >= M.n_cells) return;
    double ub[D::NC], ab[D::NA];
ABL_UNROLL_SPECIES
    for (int k = 0; k < D::NC; k++) ub[k] = __ldg(in.ub + k * M.gs + m);
ABL_UNROLL_SPECIES
    for (int k = 0; k < D::NA; k++) ab[k] = __ldg(in.ab + k * M.gs + m);
    const int beg = M.cone_ptr[m], end = M.cone_ptr[m + 1];
    const size_t wb = weight_base(M, m, beg);
    // the next entry is loaded while this neighbour's rows arrive: the pass waits for loads alone (96^3 box
    // 213 -> 201 us, 56^3 with five species 73 -> 65 us)
    int2 next = beg < end ? M.cone[beg] : make_int2(0, 0);
#pragma unroll 1
    for (int i = beg; i < end; i++) {
        const int2 ce = next;
        if (i + 1 < end) next = M.cone[i + 1];
        const int f = ce.x, n = ce.y & kConeNbr;
        double w[DIM], wa[DIM];
        cone_weights<DIM, double>(M.cwar, nullptr, wb + (size_t)(i - beg), w, wa);
        if (do_state) {
            if (!(ce.y & kConeBoundary)) {
                double gn[GC::S];
                load_comps<GC::S>(in.gb, M.gs, n, gn);
ABL_UNROLL_SPECIES
                for (int k = 0; k < D::NC; k++)
#pragma unroll
                    for (int d = 0; d < DIM; d++) ub[k] += w[d] * gn[k * DIM + d];
            }
ABL_UNROLL_SPECIES
            for (int k = 0; k < D::NC; k++)
                if (__ldg(in.fstar + k * M.gs + n) == f) ub[k] += __ldg(in.beta + k * M.gs + n);
        }
        if (do_aux) {
            double gn[GC::A];
            load_comps<GC::A>(in.gab, M.gs, n, gn);
            contract_aux<DIM, NS>(1.0, wa, gn, ab);
        }
    }
    double u[D::NC];
    load_state<DIM, NS>(U, m, u);
    cell_aux_vjp<DIM, NS>(P, u, tmp, m, ab, ub);
    bool finite = true;
ABL_UNROLL_SPECIES
    for (int k = 0; k < D::NC; k++) {
        Ub[(size_t)m * D::NC + k] += ub[k];
        finite = finite && isfinite(ub[k]);
    }
    if (!finite) atomicOr(status, kStatusNaN);
}

}  // namespace abl
