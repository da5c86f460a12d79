// Grid-side rheology kernels: strain rates, centroid<->vertex averaging, the
// local visco-elasto-plastic solve per node and phase with its consistent
// tangent, the rheological operators D11..D34 and the momentum RHS.
//
// Reference behaviour followed (paths inside the MDOODZ 6.0 repository):
//   StrainRateComponents            SOURCE/RheologyDensity.c:1902-1984
//   InterpCentroidsToVerticesDouble SOURCE/GridRoutines.c:106-198
//   InterpVerticesToCentroidsDouble SOURCE/GridRoutines.c:204-228
//   Viscosity                       SOURCE/RheologyDensity.c:44-707
//   NonNewtonianViscosityGrid       SOURCE/RheologyDensity.c:961-1415
//   RheologicalOperators            SOURCE/RheologyDensity.c:713-954
//   EvaluateRHS                     SOURCE/StokesRoutines.c:922-1133
// Isotropic, incompressible, non-reactive subset; the host rejects the rest.
#include <cmath>
#include "mdz_internal.cuh"
#include "mlp.cuh"


#define ZEROC 273.15

// ---------------------------------------------------------------------------
// Strain rates: exz at the vertices; div, exx, ezz at the centroids (one thread
// per vertex, which takes the centroid of its number too).
__global__ void k_strain(mdz_dgrid g, const double *__restrict__ u, const double *__restrict__ v,
                         double *__restrict__ div, double *__restrict__ exx, double *__restrict__ ezz,
                         double *__restrict__ exz) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, Nx = g.Nx, ncx = g.ncx;
    if (i < ncx * g.ncz) {
        const int k = i % ncx, l = i / ncx, c1 = k + l * Nx, c2 = k + l * (Nx + 1);
        const signed char t = g.BCp[i];
        double d = 0.0, ex = 0.0, ez = 0.0;
        if (t != 30 && t != 31) {
            const double dudx = (u[c1 + 1 + Nx] - u[c1 + Nx]) * g.idx, dvdz = (v[c2 + 1 + (Nx + 1)] - v[c2 + 1]) * g.idz;
            d = dudx + dvdz;
            ex = dudx - 1.0 / 3.0 * d;
            ez = dvdz - 1.0 / 3.0 * d;
        }
        div[i] = d; exx[i] = ex; ezz[i] = ez;
    }
    if (i < Nx * g.Nz) {
        const int k = i % Nx, l = i / Nx, c2 = k + l * (Nx + 1);
        double e = 0.0;
        if (g.BCg[i] != 30) {
            if (g.BCu[i] != 30 && g.BCu[i + Nx] != 30) e += 0.5 * (u[i + Nx] - u[i]) * g.idz;
            if (g.BCv[c2] != 30 && g.BCv[c2 + 1] != 30) e += 0.5 * (v[c2 + 1] - v[c2]) * g.idx;
        }
        exz[i] = e;
    }
}

// Centroid -> vertex averages of N fields with the zero-flux padding of the
// reference: the padded ring repeats the nearest interior centroid (corners:
// diagonal).  The fields share the indices and tags: seven single-field launches
// per evaluation took 54 us at 1024 x 512; in two, one of them together with the
// shear rate's average (21 us by itself), 42.
template <int N>
struct c2v_fields { const double *cen[N]; double *ver[N]; };

template <int N>
__device__ __forceinline__ void c2v(const mdz_dgrid &g, int c1, const c2v_fields<N> &F) {
    const int Nx = g.Nx, ncx = g.ncx, ncz = g.ncz, k = c1 % Nx, l = c1 / Nx;
    const bool rock = g.BCg[c1] != 30;
    // padded indices of the four centroids around vertex (k, l): columns k-1, k; rows l-1, l
    const int kw = k - 1 < 0 ? 0 : k - 1, ke = k > ncx - 1 ? ncx - 1 : k;
    const int ls = l - 1 < 0 ? 0 : l - 1, ln = l > ncz - 1 ? ncz - 1 : l;
    double r[N];
#pragma unroll
    for (int f = 0; f < N; f++) {
        const double *cen = F.cen[f];
        r[f] = rock ? 0.25 * (cen[kw + ls * ncx] + cen[ke + ls * ncx] + cen[kw + ln * ncx] + cen[ke + ln * ncx]) : 0.0;
    }
#pragma unroll
    for (int f = 0; f < N; f++) F.ver[f][c1] = r[f];
}

template <int N>
__global__ void k_c2v(mdz_dgrid g, c2v_fields<N> F) {
    const int c1 = blockIdx.x * blockDim.x + threadIdx.x;
    if (c1 < g.Nx * g.Nz) c2v<N>(g, c1, F);
}

// exz from the vertices to the centroids (mean over the rock ones), and the
// normal strain rates from the centroids to the vertices.
__global__ void k_strain_averages(mdz_dgrid g, const double *__restrict__ exz, double *__restrict__ exz_n,
                                  c2v_fields<2> F) {
    const int i = blockIdx.x * blockDim.x + threadIdx.x, Nx = g.Nx, ncx = g.ncx;
    if (i < ncx * g.ncz) {
        const int k = i % ncx, l = i / ncx, c1 = k + l * Nx;
        double e = 0.0;
        int n = 0;
        if (g.BCp[i] != 30 && g.BCp[i] != 31) {
            if (g.BCg[c1] != 30) { e += exz[c1]; n++; }
            if (g.BCg[c1 + 1] != 30) { e += exz[c1 + 1]; n++; }
            if (g.BCg[c1 + Nx] != 30) { e += exz[c1 + Nx]; n++; }
            if (g.BCg[c1 + Nx + 1] != 30) { e += exz[c1 + Nx + 1]; n++; }
            if (n == 4) e *= 0.25;   // (the quotient, without an FP64 division)
            else if (n > 0) e /= n;
        }
        exz_n[i] = e;
    }
    if (i < Nx * g.Nz) c2v<2>(g, i, F);
}

__global__ void k_v2c(mdz_dgrid g, double *__restrict__ cen, const double *__restrict__ ver) {
    int c0 = blockIdx.x * blockDim.x + threadIdx.x;
    int ncx = g.ncx, Nx = g.Nx;
    if (c0 >= ncx * g.ncz) return;
    int k = c0 % ncx, l = c0 / ncx, c1 = k + l * Nx;
    if (g.BCp[c0] != 30 && g.BCp[c0] != 31) cen[c0] = 0.25 * (ver[c1] + ver[c1 + 1] + ver[c1 + Nx] + ver[c1 + 1 + Nx]);
}

// ---------------------------------------------------------------------------
// Local solve.  Outputs of one (node, phase) solve.
struct visc_res {
    double eta, txx, tzz, txz, etaVE, VEcoeff, Eii_el, Eii_pl, Eii_pwl, Eii_lin, Eii_cst, Eii_exp, Eii_gbs;
    double Exx_el, Ezz_el, Exz_el, Exx_diss, Ezz_diss, Exz_diss, d1;
    double detadexx, detadezz, detadexz, detadp, X1, OverS;
    double ddivpdexx, ddivpdezz, ddivpdexz, ddivpdp, Pcorr, div_el, div_pl;
    double eta_ve, gdot;    // converged local unknowns (training labels of the learned guess)
    double eta_up;          // the reference's start of the visco-elastic iteration
    int ve_fail, vp_fail, ve_its, vp_its;
    int learned, fallback;  // started from a learned guess; polish failed and the plain solve reran
    float lab_x, lab_y;     // the converged solve as a start: ln(eta_ve / eta_up), gdot / (2 Eii)
};

// Polish budget of a learned start: Newton-type updates allowed before the
// plain solve takes over.
#define MDZ_POLISH_STEPS 3

// Precision-generic helpers of the local solve (FP64 or FP32 instances).
__device__ __forceinline__ double msqrt(double x) { return sqrt(x); }
__device__ __forceinline__ float msqrt(float x) { return sqrtf(x); }
__device__ __forceinline__ double mexp(double x) { return exp(x); }
__device__ __forceinline__ float mexp(float x) { return expf(x); }
__device__ __forceinline__ double mlog(double x) { return log(x); }
__device__ __forceinline__ float mlog(float x) { return logf(x); }
__device__ __forceinline__ double mfabs(double x) { return fabs(x); }
__device__ __forceinline__ float mfabs(float x) { return fabsf(x); }
__device__ __forceinline__ double msin(double x) { return sin(x); }
__device__ __forceinline__ float msin(float x) { return sinf(x); }
__device__ __forceinline__ void msincos(double x, double *s, double *c) { sincos(x, s, c); }
__device__ __forceinline__ void msincos(float x, float *s, float *c) { sincosf(x, s, c); }
__device__ __forceinline__ double mpow(double x, double y) { return pow(x, y); }
__device__ __forceinline__ float mpow(float x, float y) { return powf(x, y); }

template <typename Real>
__device__ __forceinline__ Real dmin(Real a, Real b) { return a <= b ? a : b; }

// ---- constants of the local solves, taken once per launch on the host -----------
// The local solves are bound by the FP64 pipe (77 % active): a transcendental
// function is 20-100 FP64 instructions, a division ten, and every comparison
// or conversion of an FP64 value is one too.  So whatever depends on the
// phase and the model switches alone is formed here: reciprocals, prefactors,
// powers of the reference grain size, and flags in place of comparisons.
enum {
    VP_CST = 1, VP_PWL = 2, VP_LIN = 4, VP_EXP = 8, VP_GBS = 16, VP_TENS = 32,   // mechanisms (cstv, pwlv, ...)
    VP_LOGF = 64,      // FP64 dislocation creep in log form (lnK_pwl below)
    VP_LIN1 = 128,     // n_lin = 1: linear diffusion creep
    VP_VP1 = 256,      // n_vp = 1: linear viscoplastic regularisation
    VP_PWL_D = 512, VP_PWL_PHI = 1024, VP_LIN_D = 2048, VP_LIN_PHI = 4096,   // grain size / melt exponents not 0
    VP_GBS_D = 8192, VP_GBS_PHI = 16384
};
template <typename Real>
struct visc_phase {
    int flags;
    // dislocation creep: B = K0 exp((Q + P V) in / RT) d^md exp(-a phi), K0 = pref F A^-in f^(-r in), lnK its
    // logarithm; in = 1 / n, md = m in, a = a in (the others alike)
    Real n_pwl, in_pwl, Q_pwl, V_pwl, K0_pwl, lnK_pwl, md_pwl, a_pwl;
    Real n_lin, in_lin, Q_lin, V_lin, K0_lin, m_lin, a_lin, dm_lin, dmn_lin;   // gs_ref^-m, gs_ref^(m in)
    Real n_gbs, in_gbs, Q_gbs, V_gbs, K0_gbs, md_gbs, a_gbs;
    Real Gexp, Qexp, Sexp, Eexp, nexp;
    Real eta0, ieta0, gs_ref, igs_ref, Slim, eta_vp, in_vp;
};
template <typename Real>
struct visc_prm {
    int iselastic, step, clamp_tangent;
    Real R, dt, idt, Emin, Tmin, Tpeierls, eta_big, P_tens, mineta, maxeta;
};
template <typename Real>
struct visc_mat {
    int n_phases;
    visc_prm<Real> prm;
    visc_phase<Real> ph[MDZ_MAX_PHASES];
};

// lnK_pwl = ln(pref F A^(-1/n) f^(-r/n)): the part of the logarithm of the
// dislocation prefactor B_pwl (Viscosity, SOURCE/RheologyDensity.c:153-154)
// that depends on neither the node nor the iteration; without VP_LOGF, where
// the product is not positive and finite, the solve multiplies the reference's
// factors out as they stand.
template <typename Real>
static visc_mat<Real> make_visc_mat(const mdz_materials &m, const mdz_rheo_params &prm) {
    visc_mat<Real> k{};
    k.n_phases = m.n_phases;
    visc_prm<Real> &q = k.prm;
    q.iselastic = prm.iselastic; q.step = prm.step; q.clamp_tangent = prm.clamp_tangent;
    q.R = (Real)m.R; q.dt = (Real)prm.dt; q.idt = (Real)(1.0 / prm.dt);
    q.Emin = (Real)(1e-30 / prm.scale_E); q.Tmin = (Real)(ZEROC / prm.scale_T);
    q.Tpeierls = (Real)((1200.0 + ZEROC) / prm.scale_T); q.eta_big = (Real)(1.0e100 / prm.scale_eta);
    q.P_tens = (Real)(-25e6 / prm.scale_S); q.mineta = (Real)prm.mineta; q.maxeta = (Real)prm.maxeta;
    auto prefactor = [](double pf, double A, double n, double f, double r) {
        double v = pf * std::pow(A, -1.0 / n);
        if (r != 0) v *= std::pow(f, -r / n);
        return v;
    };
    for (int p = 0; p < m.n_phases; p++) {
        visc_phase<Real> &v = k.ph[p];
        const double n = m.npwl[p], pf = m.pref_pwl[p] * m.Fpwl[p], A = m.Apwl[p], f = m.fpwl[p], r = m.rpwl[p];
        int fl = (m.cstv[p] ? VP_CST : 0) | (m.pwlv[p] ? VP_PWL : 0) | (m.linv[p] ? VP_LIN : 0) | (m.expv[p] ? VP_EXP : 0) |
                 (m.gbsv[p] ? VP_GBS : 0) | (m.is_tensile[p] ? VP_TENS : 0);
        if (m.pwlv[p]) {
            if (m.mpwl[p] != 0) fl |= VP_PWL_D;
            if (m.apwl[p] != 0) fl |= VP_PWL_PHI;
            v.n_pwl = (Real)n; v.in_pwl = (Real)(1.0 / n); v.Q_pwl = (Real)m.Qpwl[p]; v.V_pwl = (Real)m.Vpwl[p];
            v.K0_pwl = (Real)prefactor(pf, A, n, f, r);
            v.md_pwl = (Real)(m.mpwl[p] / n); v.a_pwl = (Real)(m.apwl[p] / n);
            if (sizeof(Real) == 8 && pf > 0 && A > 0 && (r == 0 || f > 0)) {
                double l = std::log(pf) - std::log(A) / n;
                if (r != 0) l -= r / n * std::log(f);
                if (std::isfinite(l)) { v.lnK_pwl = (Real)l; fl |= VP_LOGF; }
            }
        }
        if (m.linv[p]) {
            const double nl = m.nlin[p];
            if (nl == 1.0) fl |= VP_LIN1;
            if (m.mlin[p] != 0) fl |= VP_LIN_D;
            if (m.alin[p] != 0) fl |= VP_LIN_PHI;
            v.n_lin = (Real)nl; v.in_lin = (Real)(1.0 / nl); v.Q_lin = (Real)m.Qlin[p]; v.V_lin = (Real)m.Vlin[p];
            v.K0_lin = (Real)prefactor(m.Flin[p], m.Alin[p], nl, m.flin[p], m.rlin[p]);
            v.m_lin = (Real)m.mlin[p]; v.a_lin = (Real)(m.alin[p] / nl);
            v.dm_lin = (Real)(m.mlin[p] == 0 ? 1.0 : std::pow(m.gs_ref[p], -m.mlin[p]));
            v.dmn_lin = (Real)(m.mlin[p] == 0 ? 1.0 : std::pow(m.gs_ref[p], m.mlin[p] / nl));
        }
        if (m.gbsv[p]) {
            const double ng = m.ngbs[p];
            if (m.mgbs[p] != 0) fl |= VP_GBS_D;
            if (m.agbs[p] != 0) fl |= VP_GBS_PHI;
            v.n_gbs = (Real)ng; v.in_gbs = (Real)(1.0 / ng); v.Q_gbs = (Real)m.Qgbs[p]; v.V_gbs = (Real)m.Vgbs[p];
            v.K0_gbs = (Real)prefactor(m.Fgbs[p], m.Agbs[p], ng, m.fgbs[p], m.rgbs[p]);
            v.md_gbs = (Real)(m.mgbs[p] / ng); v.a_gbs = (Real)(m.agbs[p] / ng);
        }
        v.Gexp = (Real)m.Gexp[p]; v.Qexp = (Real)m.Qexp[p]; v.Sexp = (Real)m.Sexp[p]; v.Eexp = (Real)m.Eexp[p];
        v.nexp = (Real)m.nexp[p];
        v.eta0 = (Real)m.eta0[p]; v.ieta0 = (Real)(1.0 / m.eta0[p]);
        v.gs_ref = (Real)m.gs_ref[p]; v.igs_ref = (Real)(1.0 / m.gs_ref[p]);
        v.Slim = (Real)m.Slim[p]; v.eta_vp = (Real)m.eta_vp[p]; v.in_vp = (Real)(1.0 / m.n_vp[p]);
        if (m.n_vp[p] == 1.0) fl |= VP_VP1;
        v.flags = fl;
    }
    return k;
}

// ln(1 + x) by its Mercator series through x^7, for |x| < 1/32 (truncation
// below x^8 / 8 < 2^-43): the Halley update of the learned start needs only
// its root at x = 0 to be exact, and the FP64 logarithm costs several times
// these seven multiply-adds on this part.
__device__ __forceinline__ double ln1p_series(double x) {
    return x * (1.0 + x * (-0.5 + x * (1.0 / 3.0 + x * (-0.25 + x * (0.2 + x * (-1.0 / 6.0 + x * (1.0 / 7.0)))))));
}

// ln(1 + x) to rounding, for |x| < 1/32: its Mercator series through x^11 (the
// rest is below x^12 / 12 < 2^-63).
__device__ __forceinline__ double ln1p_small(double x) {
    double p = 1.0 / 11.0;
    p = -0.1 + x * p;
    p = 1.0 / 9.0 + x * p;
    p = -0.125 + x * p;
    p = 1.0 / 7.0 + x * p;
    p = -1.0 / 6.0 + x * p;
    p = 0.2 + x * p;
    p = -0.25 + x * p;
    p = 1.0 / 3.0 + x * p;
    p = -0.5 + x * p;
    return x + x * (x * p);
}

// One (node, phase) solve.  The reference's Gxx.. (rates with the anisotropic
// elastic correction) equal Exx.. in this isotropic subset, and its f_ani =
// Gii / Eii is 1.  ie: 1 / (mu dt) where the model is elastic.
template <typename Real>
__device__ void visc_local_t(const visc_phase<Real> &m, const visc_prm<Real> &prm, Real G, Real ie, Real T, Real P,
                             Real d, Real phi, Real X0, Real Exx, Real Ezz, Real Exz, Real Txx0, Real Tzz0, Real Txz0,
                             Real dil, Real fric, Real C, Real P0, Real beta, visc_res &o, const float *guess) {
    const Real dt = prm.dt, tol = sizeof(Real) == 8 ? Real(1.0e-11) : Real(1.0e-4);
    const int nitmax = 20, fl = m.flags;
    // FP64 reports what the reference's own test after its loops (:417, :529) stops on: the last
    // iteration's convergence, not a loop that ran out.  In FP32 a failure means the FP64 solve takes
    // over, which is for every loop that ran out above the tolerance.
    constexpr bool EXHAUSTED = sizeof(Real) == 4;
    int it;
    const bool elastic = prm.iselastic != 0 && prm.step != 0;
    const bool constant = fl & VP_CST, dislocation = fl & VP_PWL, diffusion = fl & VP_LIN, lin1 = fl & VP_LIN1,
               vp1 = fl & VP_VP1, logform = sizeof(Real) == 8 && (fl & VP_LOGF);
    // Peierls creep only below 1200 C (tested before the 0 C clamp, :137),
    // grain-boundary sliding, tension cut-off; the learned start models none
    // of them, so their solves take the reference's start
    const bool peierls = (fl & VP_EXP) && T < prm.Tpeierls, gbs = fl & VP_GBS, tensile = fl & VP_TENS;
    if (peierls || gbs || tensile) guess = nullptr;
    Real res = Real(0.0);
    const Real Tii0 = msqrt(Txx0 * Txx0 + Txz0 * Txz0);
    const Real n_pwl = m.n_pwl, n_lin = m.n_lin;
    Real C_pwl = 0, C_lin = 0;
    Real eta_pwl = Real(0.0), eta_lin = Real(0.0), eta_vep = Real(0.0), eta_vp = Real(0.0);
    const Real eta_vp0 = m.eta_vp;
    Real Eii_pwl = 0, Eii_lin = 0, Eii_cst = 0, Eii_exp = 0, Eii_gbs = 0;
    o.Eii_pl = Real(0.0); o.OverS = Real(0.0); o.ve_fail = 0; o.vp_fail = 0; o.vp_its = 0;

    const Real Eyy = -(Exx + Ezz);
    Real Eii = msqrt(Real(0.5) * (Exx * Exx + Ezz * Ezz + Eyy * Eyy) + Exz * Exz);
    if (Eii < prm.Emin) Eii = prm.Emin;
    const Real iEii = Real(1.0) / Eii;
    o.Pcorr = P;
    o.d1 = m.gs_ref;
    // without elasticity the reference sets G = K = 10 and no dilation
    if (!elastic) { G = Real(1e1); dil = Real(0.0); }
    const Real eta_el = G * dt;
    const Real i2eta_el = Real(0.5) * (elastic && prm.iselastic == 1 ? ie : Real(1.0) / eta_el);
    if (T < prm.Tmin) T = prm.Tmin;
    const Real iRT = Real(1.0) / (prm.R * T);
    // FP64 dislocation creep in log form: ln B_pwl from the per-phase constant,
    // then C_pwl = (2 B_pwl)^-n and eta_pwl = B_pwl Eii^(1/n - 1) as two
    // exponentials after one logarithm (the product form takes three pow and an
    // exp), and in the iterations Eii_pwl = exp(ln C_pwl + n ln Tii) with
    // ln Tii = lnTE + ln eta_ve.  FP32 keeps the product form: rounding of
    // the logarithms' sums there is at the size of its convergence test.
    Real lnC_pwl = Real(0.0), lnTE = Real(0.0), ln_eta_pwl = Real(0.0);
    if (dislocation) {
        const Real in = m.in_pwl;
        if (logform) {
            Real lnB = m.lnK_pwl + (m.Q_pwl + P * m.V_pwl) * iRT * in;
            if (fl & VP_PWL_D) lnB += m.md_pwl * mlog(d);
            if (fl & VP_PWL_PHI) lnB -= m.a_pwl * phi;
            const Real ln2 = Real(0.69314718055994530942), LE = mlog(Eii);
            lnTE = ln2 + LE;   // ln(2 Eii) = ln Tii - ln eta_ve
            lnC_pwl = -n_pwl * (ln2 + lnB);
            C_pwl = mexp(lnC_pwl);
            ln_eta_pwl = lnB + (in - Real(1.0)) * LE;
            eta_pwl = mexp(ln_eta_pwl);
        } else {
            Real B_pwl = m.K0_pwl * mexp((m.Q_pwl + P * m.V_pwl) * iRT * in);
            if (fl & VP_PWL_D) B_pwl *= mpow(d, m.md_pwl);
            if (fl & VP_PWL_PHI) B_pwl *= mexp(-m.a_pwl * phi);
            C_pwl = mpow(Real(2.0) * B_pwl, -n_pwl);
            eta_pwl = B_pwl * mpow(Eii, in - Real(1.0));
        }
    }
    Real B_lin = 0;
    if (diffusion) {
        B_lin = m.K0_lin * mexp((m.Q_lin + P * m.V_lin) * iRT * m.in_lin);
        if (fl & VP_LIN_PHI) B_lin *= mexp(-m.a_lin * phi);
        C_lin = lin1 ? Real(0.5) / B_lin : mpow(Real(2.0) * B_lin, -n_lin);
        eta_lin = lin1 ? B_lin : B_lin * mpow(Eii, m.in_lin - Real(1.0));
        if (fl & VP_LIN_D) eta_lin *= mpow(d, m.m_lin * m.in_lin);
    }
    // grain-boundary sliding: a creep law of the dislocation form (:176-180)
    Real C_gbs = Real(0.0), eta_gbs = Real(0.0);
    if (gbs) {
        Real B_gbs = m.K0_gbs * mexp((m.Q_gbs + P * m.V_gbs) * iRT * m.in_gbs);
        if (fl & VP_GBS_D) B_gbs *= mpow(d, m.md_gbs);
        if (fl & VP_GBS_PHI) B_gbs *= mexp(-m.a_gbs * phi);
        C_gbs = mpow(Real(2.0) * B_gbs, -m.n_gbs);
        eta_gbs = B_gbs * mpow(Eii, m.in_gbs - Real(1.0));
    }
    // Peierls creep, exponential law as a power law of exponent ST + n
    // (:181-199): ST = Q / RT 2 gamma (1 - gamma)
    const Real n_exp = m.nexp;
    Real ST = Real(0.0), B_exp = Real(0.0), C_exp = Real(0.0), eta_exp = Real(0.0);
    if (peierls) {
        const Real gam = m.Gexp, Ea = m.Qexp;
        ST = Ea * iRT * Real(2.0) * gam * (Real(1.0) - gam);
        const Real sn = ST + n_exp, isn = Real(1.0) / sn;
        const Real Arr = mexp(-Ea * iRT * (Real(1.0) - gam) * (Real(1.0) - gam));
        const Real F_exp = mpow(mpow(Real(2.0), Real(1.0) - ST - n_exp) / mpow(msqrt(Real(3.0)), sn + Real(1.0)), isn);
        B_exp = F_exp * (mpow(gam * m.Sexp, ST * isn) / mpow(m.Eexp * Arr, isn));
        C_exp = mpow(Real(2.0) * B_exp, -sn);
        eta_exp = B_exp * mpow(Eii, isn - Real(1.0));
    }
    Real cos_fric, sin_fric;
    msincos(fric, &sin_fric, &cos_fric);
    Real sin_dil = dil == Real(0.0) ? Real(0.0) : msin(dil);
    Real Tyield = C * cos_fric + P * sin_fric;
    if (m.Slim < Tyield) { sin_fric = Real(0.0); cos_fric = Real(1.0); sin_dil = Real(0.0); C = m.Slim; Tyield = m.Slim; }
    // tension cut-off (:204-213): below the tension pressure -25 MPa the yield
    // line turns to pass through (P_tens, 0)
    bool tens = false;
    if (tensile) {
        const Real sin_fric_tens = -C * cos_fric / prm.P_tens;
        if (C * cos_fric + P * sin_fric_tens < Tyield) {
            sin_fric = sin_fric_tens;
            Tyield = C * cos_fric + P * sin_fric_tens;
            tens = true;
        }
    }
    o.X1 = X0;
    Real eta_up = prm.eta_big;
    if (constant) eta_up = dmin(eta_up, m.eta0);
    if (dislocation) eta_up = dmin(eta_up, eta_pwl);
    if (elastic) eta_up = dmin(eta_up, eta_el);
    if (peierls) eta_up = dmin(eta_up, eta_exp);
    if (diffusion) eta_up = dmin(eta_up, eta_lin);
    if (gbs) eta_up = dmin(eta_up, eta_gbs);
    // local Newton on the visco-elastic viscosity
    Real eta_ve = eta_up, Tii;
    const Real dm_lin = m.dm_lin;
    bool ve_done = false;
    o.eta_up = eta_up;
    o.learned = guess != nullptr;
    o.fallback = 0;
    const Real ifcst = constant ? Real(0.5) * m.ieta0 : Real(0.0), iel = elastic ? i2eta_el : Real(0.0);
    // logarithm of the start, known where dislocation creep sets it
    const bool start_pwl = logform && eta_up == eta_pwl;
    if (guess) {
        // Learned start s = mlog(eta_ve), polished by Halley steps on
        // g(s) = mlog(sum of the strain rates) - mlog(Eii): every mechanism's
        // rate is c_k mexp(n_k s), so g' and g'' are rate-weighted means of n_k
        // and n_k^2 (in s the residual is nearly linear; Halley in eta itself
        // left 39 % of the solves unconverged after two steps).  Converged
        // means the reference's own test below holds.  The network predicts
        // ln(eta_ve / eta_up), eta_up being the reference's start (the
        // smallest viscosity of the active mechanisms).
        Real s = (start_pwl ? ln_eta_pwl : mlog(eta_up)) + (Real)guess[0];
        for (it = 0; it <= MDZ_POLISH_STEPS; it++) {
            eta_ve = mexp(s);
            Tii = Real(2.0) * eta_ve * Eii;
            const Real Eel = Tii * iel;
            Eii_cst = Tii * ifcst;
            if (dislocation) Eii_pwl = logform ? mexp(lnC_pwl + n_pwl * (lnTE + s)) : C_pwl * mpow(Tii, n_pwl);
            if (diffusion) Eii_lin = C_lin * (lin1 ? Tii : mpow(Tii, n_lin)) * dm_lin;
            const Real S0 = Eel + Eii_pwl + Eii_lin + Eii_cst;
            res = mfabs((Eii - S0) * iEii);
            // a start is accepted only after one update: a warm start can
            // pass the test as it stands, with an error the size of the change
            // in strain rate since it was recorded (the reference's iteration
            // always ends one quadratic step past the test)
            if (it > 0 && res < tol / 100) { ve_done = true; break; }
            if (it == MDZ_POLISH_STEPS) break;
            if (!(S0 > Real(0.0))) break;
            const Real E1 = n_pwl * Eii_pwl, E2 = lin1 ? Eii_lin : n_lin * Eii_lin;
            const Real S1 = Eel + E1 + E2 + Eii_cst;
            const Real S2 = Eel + n_pwl * E1 + (lin1 ? E2 : n_lin * E2) + Eii_cst;
            const Real iS0 = Real(1.0) / S0;
            const Real q = S0 * iEii;
            const Real g = (sizeof(Real) == 8 && mfabs(q - Real(1.0)) < Real(0.03125)) ? Real(ln1p_series(double(q - Real(1.0)))) : mlog(q);
            const Real g1 = S1 * iS0, g2 = S2 * iS0 - g1 * g1;
            const Real den = Real(2.0) * g1 * g1 - g * g2;
            s -= den > Real(0.0) ? Real(2.0) * g * g1 / den : g / g1;
        }
        o.ve_its = it;
        if (!ve_done) {
            o.fallback = 1;
            eta_ve = eta_up;
            Eii_pwl = 0; Eii_lin = 0; Eii_cst = 0;
        }
    }
    // the reference's Newton iteration, eta_ve -= r / f', with f' multiplied by
    // eta_ve.  The log form needs ln eta_ve: known at the start where dislocation
    // creep sets it, then moved by ln(1 - x) for a relative change x, by its series
    // (13 FP64 instructions, the logarithm 29) once |x| < 1/32, as in the last
    // two or three of some five iterations: 513 x 257 centroids 219 -> 207 us.  The
    // sums round at 1e-16 each, the logarithm of a viscosity at half a unit of some 50.
    // Not beside grain-boundary sliding: the reference's f' leaves it out, so an update
    // may overshoot to a negative viscosity, which has no logarithm but, at integer
    // exponents, has the power.  (Without it S is convex and the iteration comes
    // down on the root from above.)
    const Real dfl = -Real(2.0) * Eii * (iel + ifcst);
    const bool log_it = logform && dislocation && !gbs;
    Real ln_eta = Real(0.0);
    if (log_it && !ve_done) ln_eta = eta_ve == eta_up && start_pwl ? ln_eta_pwl : mlog(eta_ve);
    for (it = 0; !ve_done && it < nitmax; it++) {
        Tii = Real(2.0) * eta_ve * Eii;
        Eii_cst = Tii * ifcst;
        if (dislocation) {
            if (log_it) Eii_pwl = mexp(lnC_pwl + n_pwl * (lnTE + ln_eta));
            else Eii_pwl = C_pwl * mpow(Tii, n_pwl);
        }
        if (gbs) Eii_gbs = C_gbs * mpow(Tii, m.n_gbs);
        if (peierls) Eii_exp = C_exp * mpow(Tii, ST + n_exp);
        if (diffusion) Eii_lin = C_lin * (lin1 ? Tii : mpow(Tii, n_lin)) * dm_lin;
        const Real r = Eii - Tii * iel - (Eii_pwl + Eii_exp + Eii_lin + Eii_gbs + Eii_cst);
        res = mfabs(r * iEii);
        if (res < tol / 100) break;
        // (grain-boundary sliding has no term here in the reference)
        Real S1 = (lin1 ? Eii_lin : Eii_lin * n_lin) + Eii_pwl * n_pwl;
        if (peierls) S1 += Eii_exp * (ST + n_exp);
        const Real x = r / (dfl * eta_ve - S1);
        eta_ve -= x * eta_ve;
        if (log_it) {
            if (mfabs(x) < Real(0.03125)) ln_eta += Real(ln1p_small(double(-x)));
            else ln_eta = mlog(eta_ve);
        }
    }
    if (!ve_done) {   // iterations of a failed polish count too
        o.ve_its = it + (guess ? MDZ_POLISH_STEPS : 0);
        if (EXHAUSTED ? it == nitmax && !(res <= tol) : it == nitmax - 1 && res > tol) o.ve_fail = 1;
    }
    o.eta_ve = eta_ve;
    // the rates were evaluated at the final eta_ve when the iteration stopped
    // on its convergence test (not when it ran out): viscosities and powers of
    // Tii below then follow from them, eta_k = Tii / (2 Eii_k) and
    // C_pwl Tii^n = Eii_pwl, without another FP64 pow each
    const bool fresh = ve_done || res < tol / 100;
    Tii = Real(2.0) * eta_ve * Eii;
    if (dislocation && !fresh) Eii_pwl = C_pwl * mpow(Tii, n_pwl);
    const Real iTii = Real(1.0) / Tii, two_eta = Real(2.0) * eta_ve;   // Tii / Eii
    Real Txx = Exx * two_eta, Tzz = Ezz * two_eta, Txz = Exz * two_eta;
    Real Exx_lin = 0, Ezz_lin = 0, Exz_lin = 0, Exx_cst = 0, Ezz_cst = 0, Exz_cst = 0;
    Real Exx_exp = 0, Ezz_exp = 0, Exz_exp = 0;
    Real inv_eta_diss = Real(0.0);
    if (peierls) {
        eta_exp = B_exp * mpow(Eii_exp, Real(1.0) / (ST + n_exp) - Real(1.0));
        const Real h = Real(0.5) / eta_exp;
        inv_eta_diss += Real(2.0) * h;
        Exx_exp = Txx * h; Ezz_exp = Tzz * h; Exz_exp = Txz * h;
    }
    Real h_pwl = Eii_pwl * iTii;   // 1 / (2 eta_pwl) = C_pwl Tii^(n-1)
    if (dislocation) inv_eta_diss += Real(2.0) * h_pwl;
    if (diffusion) {
        const Real h = fresh ? Eii_lin * iTii
                             : Real(0.5) / (B_lin * (lin1 ? Real(1.0) : mpow(Eii_lin, m.in_lin - Real(1.0))) * m.dmn_lin);
        inv_eta_diss += Real(2.0) * h;
        Exx_lin = Txx * h; Ezz_lin = Tzz * h; Exz_lin = Txz * h;
    }
    if (constant) {
        const Real h = Real(0.5) * m.ieta0;
        inv_eta_diss += m.ieta0;
        Exx_cst = Txx * h; Ezz_cst = Tzz * h; Exz_cst = Txz * h;
    }
    // visco-elastic tangent
    Real deta = Real(0.0);
    if (dislocation) deta += -(Eii_pwl * iTii * iTii * iTii) * (n_pwl - Real(1.0));   // C Tii^(n-3)
    if (peierls) deta += -C_exp * mpow(Tii, n_exp + ST - Real(3.0)) * (n_exp + ST - Real(1.0));
    if (diffusion && !lin1) deta += -C_lin * mpow(Tii, n_lin - Real(3.0)) * (n_lin - Real(1.0)) * dm_lin;
    const Real e2 = eta_ve * eta_ve, de2 = deta * e2;
    const Real dTxx = de2 * (Real(2.0) * Txx + Tzz), dTzz = de2 * (Real(2.0) * Tzz + Txx), dTxz = Real(2.0) * de2 * Txz;
    const Real den = Real(1.0) - Real(2.0) * (dTxx * Exx + dTzz * Ezz + dTxz * Exz);
    const Real e2den = two_eta / den;
    const Real dve_dExx = dTxx * e2den, dve_dEzz = dTzz * e2den, dve_dExz = dTxz * e2den;
    Real dummy = Real(0.0);
    if (dislocation) dummy += Real(2.0) * h_pwl * m.V_pwl * iRT;   // -2 Tii^(n-1) dC/dP, dC/dP = -C V / RT
    if (diffusion && m.V_lin != Real(0.0)) {
        Real t = Real(2.0) * C_lin * m.V_lin * iRT;
        if (!lin1) t *= mpow(Tii, n_lin - Real(1.0));
        if (fl & VP_LIN_D) t *= mpow(d, -m.m_lin);
        dummy += t;
    }
    const Real dve_dP = e2 * dummy;
    // plastic return mapping on gdot
    Real gdot = Real(0.0), dQdtxx = 0, dQdtzz = 0, dQdtxz = 0, dQdP = 0, divp = Real(0.0), Pc = P;
    Real dlamdExx = 0, dlamdEzz = 0, dlamdExz = 0, dlamdP = 0;
    Real dvep_dExx = 0, dvep_dEzz = 0, dvep_dExz = 0, dvep_dP = 0;
    Real F_trial = Tii - Tyield;
    const bool is_pl = F_trial > Real(1e-17);
    Real Kdt = Real(0.0);
    if (is_pl || tens) Kdt = elastic ? dt / beta : Real(1e1) * dt;
    // tensile domain: the dilation angle that returns the stress to the
    // tension corner (:456-465, SimpleYields.m of the reference)
    if (tens) {
        eta_vp = vp1 ? eta_vp0 : eta_vp0 * mpow(Eii, m.in_vp - Real(1.0));
        const Real Pc_chk = -(C * cos_fric) / (-Tii / P + sin_fric);
        sin_dil = (P * eta_ve + P * eta_vp - Pc_chk * eta_ve - Pc_chk * eta_vp) /
                  (Kdt * (C * cos_fric + Pc_chk * sin_fric - Tii));
    }
    Real dsdExx = Real(0.0), dsdEzz = Real(0.0), dsdExz = Real(0.0), dsdP = Real(0.0);   // d sin_dil / d .
    if (is_pl) {
        const Real in_vp = m.in_vp, Kss = Kdt * sin_fric * sin_dil, Ccf = C * cos_fric;
        eta_vp = vp1 ? eta_vp0 : eta_vp0 * mpow(Eii, in_vp - Real(1.0));
        gdot = F_trial / (eta_ve + eta_vp + Kss);
        const Real hT = Real(0.5) * iTii;
        dQdtxx = Txx * hT; dQdtzz = Tzz * hT; dQdtxz = Txz * iTii;
        const Real tol0 = tol * F_trial;   // |F| / F_trial0 < tol
        dQdP = -sin_dil;
        bool vp_done = false;
        auto eval = [&]() {   // F at gdot (Pc, eta_vp, Tyield)
            divp = gdot * sin_dil;
            Pc = P + Kdt * divp;
            if (!vp1) eta_vp = eta_vp0 * mpow(mfabs(gdot), in_vp - Real(1.0));
            Tyield = Ccf + Pc * sin_fric + gdot * eta_vp;
            F_trial = Tii - eta_ve * gdot - Tyield;
            res = mfabs(F_trial);
            return res < tol || res < tol0;
        };
        if (guess) {
            // learned start: gdot = fraction * 2 Eii, at most MDZ_POLISH_STEPS
            // Newton updates, the reference's own convergence test
            Real frac = (Real)guess[1];
            frac = frac > Real(1e-6) ? (frac < Real(1.0) ? frac : Real(1.0)) : Real(1e-6);
            const Real gdot_plain = gdot;
            gdot = frac * Real(2.0) * Eii;
            for (it = 0; it <= MDZ_POLISH_STEPS; it++) {
                const bool ok = eval();
                if (it > 0 && ok) { vp_done = true; break; }
                if (it == MDZ_POLISH_STEPS) break;
                gdot += F_trial / (eta_ve + eta_vp * in_vp + Kss);
            }
            o.vp_its = it;
            if (!vp_done) {
                o.fallback = 1;
                gdot = gdot_plain;
            }
        }
        for (it = 0; !vp_done && it < nitmax; it++) {
            if (eval()) break;
            gdot += F_trial / (eta_ve + eta_vp * in_vp + Kss);
        }
        if (!vp_done) {
            o.vp_its = it + (guess ? MDZ_POLISH_STEPS : 0);
            if (EXHAUSTED ? it == nitmax && !(res <= tol || res <= tol0)
                          : it == nitmax - 1 && (res > tol || res > tol0)) o.vp_fail = 1;
        }
        Txx = two_eta * (Exx - gdot * dQdtxx);
        Tzz = two_eta * (Ezz - gdot * dQdtzz);
        const Real Tyy = -(Txx + Tzz);
        Txz = two_eta * (Exz - gdot * dQdtxz * Real(0.5));
        Tii = msqrt(Real(0.5) * (Txx * Txx + Tzz * Tzz + Tyy * Tyy) + Txz * Txz);
        eta_vep = Tii * Real(0.5) * iEii;
        o.Eii_pl = gdot * Real(0.5);
        o.OverS = eta_vp * gdot;
        o.Pcorr = Pc;
        // visco-elasto-plastic tangent
        if (tens) {   // derivatives of the tensile dilation angle (:578-587)
            const Real dEii_dExx = (Real(2.0) * Exx + Ezz) * Real(0.5) * iEii, dEii_dEzz = (Real(2.0) * Ezz + Exx) * Real(0.5) * iEii;
            const Real dEii_dExz = Exz * iEii;
            const Real A = Real(2.0) * Eii * eta_ve - P * sin_fric, A2 = A * A;
            const Real iden = Real(1.0) / (Kdt * A * (C * P * cos_fric * sin_fric + (Ccf - Real(2.0) * Eii * eta_ve) * A));
            const Real Q = C * P * cos_fric * sin_fric + A2;
            auto dsd = [&](Real dve, Real dE) {
                const Real dT = Eii * dve + dE * eta_ve;
                return (Real(2.0) * Kdt * sin_dil * dT * Q +
                        P * (-Ccf * dve * A + Real(2.0) * Ccf * (eta_ve + eta_vp) * dT + dve * A2)) * iden;
            };
            dsdExx = dsd(dve_dExx, dEii_dExx);
            dsdEzz = dsd(dve_dEzz, dEii_dEzz);
            dsdExz = dsd(dve_dExz, dEii_dExz);
            dsdP = (Real(2.0) * C * Eii * cos_fric * (eta_ve + eta_vp) * (P * dve_dP - eta_ve) - C * P * cos_fric * dve_dP * A +
                    Real(2.0) * Eii * Kdt * sin_dil * (C * cos_fric * sin_fric * (P * dve_dP - eta_ve) + dve_dP * A2) +
                    A2 * (P * dve_dP + eta_ve + eta_vp)) * iden;
        }
        const Real ev = eta_ve * iEii, E2 = Real(2.0) * Eii, Ksf = Kdt * sin_fric;
        const Real xx2 = Real(2.0) * Exx + Ezz, zz2 = Real(2.0) * Ezz + Exx;
        const Real gg = Real(1.0) / (eta_ve + eta_vp * in_vp + Kss);
        dlamdExx = gg * (xx2 * ev + E2 * dve_dExx - gdot * (dve_dExx + Ksf * dsdExx));
        dlamdEzz = gg * (zz2 * ev + E2 * dve_dEzz - gdot * (dve_dEzz + Ksf * dsdEzz));
        dlamdExz = gg * (Real(2.0) * Exz * ev + E2 * dve_dExz - gdot * (dve_dExz + Ksf * dsdExz));
        dlamdP = gg * (-sin_fric + E2 * dve_dP - gdot * (dve_dP + Ksf * dsdP));
        Real dvp_dExx = 0, dvp_dEzz = 0, dvp_dExz = 0, dvp_dP = 0;   // (linear regularisation: constant eta_vp)
        if (!vp1) {
            const Real evq = eta_vp / gdot * (in_vp - Real(1.0));
            dvp_dExx = evq * dlamdExx; dvp_dEzz = evq * dlamdEzz;
            dvp_dExz = evq * dlamdExz; dvp_dP = evq * dlamdP;
        }
        const Real a = eta_vp + Kss;
        const Real h2 = Real(0.5) * iEii, TyE3 = Tyield * h2 * iEii * iEii;   // 1 / (2 Eii), Tyield / (2 Eii^3)
        dvep_dExx = -Real(0.5) * xx2 * TyE3 + (a * dlamdExx + gdot * (dvp_dExx + Ksf * dsdExx)) * h2;
        dvep_dEzz = -Real(0.5) * zz2 * TyE3 + (a * dlamdEzz + gdot * (dvp_dEzz + Ksf * dsdEzz)) * h2;
        dvep_dExz = -Exz * TyE3 + (a * dlamdExz + gdot * (dvp_dExz + Ksf * dsdExz)) * h2;
        dvep_dP = (sin_fric + a * dlamdP + gdot * (dvp_dP + Ksf * dsdP)) * h2;
    }
    o.gdot = gdot;
    if (!is_pl) {
        o.detadexx = dve_dExx; o.detadezz = dve_dEzz; o.detadexz = dve_dExz; o.detadp = dve_dP;
        o.etaVE = eta_ve;
        o.ddivpdexx = Real(0.0); o.ddivpdezz = Real(0.0); o.ddivpdexz = Real(0.0); o.ddivpdp = Real(0.0);
    } else {
        o.detadexx = dvep_dExx; o.detadezz = dvep_dEzz; o.detadexz = dvep_dExz; o.detadp = dvep_dP;
        o.etaVE = eta_vep;
        o.ddivpdexx = -dQdP * dlamdExx + gdot * dsdExx;
        o.ddivpdezz = -dQdP * dlamdEzz + gdot * dsdEzz;
        o.ddivpdexz = -dQdP * dlamdExz + gdot * dsdExz;
        o.ddivpdp = -dQdP * dlamdP + gdot * dsdP;
        inv_eta_diss += Real(1.0) / eta_vep;
        // the dislocation parts of the reported rates are taken at the returned stress
        if (dislocation)
            h_pwl = !(C_pwl > Real(0.0)) ? Real(0.0)
                  : logform ? mexp(lnC_pwl + (n_pwl - Real(1.0)) * mlog(Tii)) : C_pwl * mpow(Tii, n_pwl - Real(1.0));
    }
    o.Exx_el = elastic ? (Txx - Txx0) * i2eta_el : Real(0.0);
    o.Ezz_el = elastic ? (Tzz - Tzz0) * i2eta_el : Real(0.0);
    o.Exz_el = elastic ? (Txz - Txz0) * i2eta_el : Real(0.0);
    o.Exx_diss = gdot * dQdtxx + Exx_lin + Txx * h_pwl + Exx_exp + Exx_cst;
    o.Ezz_diss = gdot * dQdtzz + Ezz_lin + Tzz * h_pwl + Ezz_exp + Ezz_cst;
    o.Exz_diss = gdot * dQdtxz * Real(0.5) + Exz_lin + Txz * h_pwl + Exz_exp + Exz_cst;
    o.Eii_el = elastic ? mfabs(Tii - Tii0) * i2eta_el : Real(0.0);
    o.Eii_pwl = Tii * h_pwl;
    o.Eii_lin = Eii_lin;
    o.Eii_cst = Eii_cst;
    o.Eii_exp = Eii_exp;
    o.Eii_gbs = Eii_gbs;
    o.div_pl = divp;
    o.div_el = -(Pc - P0) * (elastic ? beta * prm.idt : Real(0.1) * prm.idt);
    Real eta = Real(1.0) / inv_eta_diss;
    o.VEcoeff = elastic ? two_eta * i2eta_el : Real(0.0);
    if (prm.step == 0) o.etaVE = eta;
    o.txx = Txx; o.tzz = Tzz; o.txz = Txz;
    if (eta > prm.maxeta) eta = prm.maxeta;
    if (eta < prm.mineta) eta = prm.mineta;
    const bool clamped = o.etaVE > prm.maxeta || o.etaVE < prm.mineta;
    if (o.etaVE > prm.maxeta) o.etaVE = prm.maxeta;
    if (o.etaVE < prm.mineta) o.etaVE = prm.mineta;
    if (clamped && prm.clamp_tangent) {   // the limiter is flat: its tangent is zero
        o.detadexx = Real(0.0); o.detadezz = Real(0.0); o.detadexz = Real(0.0); o.detadp = Real(0.0);
    }
    o.eta = eta;
    // the start the next evaluation of this (node, phase) can polish from, in
    // the learned guess's encoding; FP32 logarithms suffice for a start
    o.lab_x = logf((float)eta_ve) - logf((float)o.eta_up);
    o.lab_y = (float)(gdot * Real(0.5) * iEii);
}

// Materials of a launch: FP64, and FP32 for the inexact evaluations.
template <bool FP32>
struct visc_mats {
    visc_mat<double> d;
    visc_mat<float> f;
};
template <>
struct visc_mats<false> {
    visc_mat<double> d;
};

// One (node, phase) local solve: in FP32 when asked (an inexact evaluation
// for a non-linear iteration far from convergence; FP64 transcendental
// functions issue at a small fraction of the FP32 rate on this part), with
// the FP64 solve taking over wherever the FP32 one failed or overflowed;
// otherwise the FP64 solve, from the learned start when one is given.
template <bool FP32>
__device__ __forceinline__ void visc_node_phase(const visc_mats<FP32> &m, int p, double G, double ie, double T, double P,
                                                double d, double phi, double X0, const double *E, double Txx0,
                                                double Tzz0, double Txz0, double dil, double fric, double C, double P0,
                                                double beta, visc_res &o, const float *guess) {
    if constexpr (FP32) {
        visc_local_t<float>(m.f.ph[p], m.f.prm, (float)G, (float)ie, (float)T, (float)P, (float)d, (float)phi, (float)X0,
                            (float)E[0], (float)E[1], (float)E[2], (float)Txx0, (float)Tzz0, (float)Txz0, (float)dil,
                            (float)fric, (float)C, (float)P0, (float)beta, o, nullptr);
        const bool ok = !o.ve_fail && !o.vp_fail && isfinite(o.eta) && isfinite(o.etaVE) && isfinite(o.txx) &&
                        isfinite(o.tzz) && isfinite(o.txz) && isfinite(o.detadexx) && isfinite(o.detadezz) &&
                        isfinite(o.detadexz) && isfinite(o.detadp) && isfinite(o.Pcorr);
        if (ok) return;
    }
    visc_local_t<double>(m.d.ph[p], m.d.prm, G, ie, T, P, d, phi, X0, E[0], E[1], E[2], Txx0, Tzz0, Txz0, dil, fric, C,
                         P0, beta, o, guess);
}

// Effective rates entering the local solve (isotropic form of the elastic
// stress correction, NonNewtonianViscosityGrid :1060-1094): E[0..2] Exx, Ezz,
// Exz and E[3..5] Gxx, Gzz, Gxz, with the reference's inverse of Da evaluated
// for ani = 0 (iDa11 = iDa22 = 1/2, iDa33 = 1, off-diagonals 0), where the two
// agree; ie = 1 / (mu dt) of an elastic model, 1 otherwise.
__device__ __forceinline__ void eff_rates(double exx, double ezz, double exz, double sxx0, double szz0, double sxz0,
                                          double ie, double *E) {
    const double h = 0.5 * ie, Exz = exz + sxz0 * h;
    E[0] = exx + sxx0 * h; E[1] = ezz + szz0 * h; E[2] = Exz;
    E[3] = E[0]; E[4] = E[1]; E[5] = Exz;
}

__device__ __forceinline__ void put(double *p, int i, double v) {
    if (p) p[i] = v;
}

// Counters of the local solves: [0] not converged, [1] learned starts whose
// polish failed (plain solve rerun), [2] learned starts (int32), and at int
// offset 48 the 64-bit total of local Newton iterations (visco-elastic plus
// plastic); warp-aggregated atomics.
__device__ __forceinline__ void count_local(int *counters, int fails, int fallbacks, int learned, int iters) {
    if (!counters) return;
    const unsigned mask = __activemask();
    const int lane = threadIdx.x & 31, leader = __ffs(mask) - 1;
    const int a = __reduce_add_sync(mask, fails), b = __reduce_add_sync(mask, fallbacks),
              c = __reduce_add_sync(mask, learned), d = __reduce_add_sync(mask, iters);
    if (lane == leader) {
        if (a) atomicAdd(&counters[0], a);
        if (b) atomicAdd(&counters[1], b);
        if (c) atomicAdd(&counters[2], c);
        if (d) atomicAdd(reinterpret_cast<unsigned long long *>(counters + 48), (unsigned long long)d);
    }
}

// One thread per centroid: loop over phases with a fraction above 1e-13.
template <bool FP32>
__global__ void __launch_bounds__(128) k_viscosity_centroids(mdz_dgrid g, const __grid_constant__ visc_mats<FP32> m,
                                                             mdz_rheo_params prm,
                                                             mdz_fields f, int *__restrict__ counters,
                                                             const float2 *guess, float2 *labels) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    int nc = g.ncx * g.ncz;
    if (c >= nc) return;
    const int avg = prm.eta_avg, nph = m.d.n_phases;
    double eta = 0, eta_phys = 0, VE = 0, sxx = 0, szz = 0, sxz = 0, eel = 0, epl = 0, epwl = 0, elin = 0, ecst = 0,
           eexp = 0, egbs = 0,
           dn = 0, xel = 0, xdi = 0, zel = 0, zdi = 0, dexx = 0, dezz = 0, dgxz = 0, dp = 0, vxx = 0, vzz = 0,
           vxz = 0, vp = 0, pc = 0, del = 0, dpl = 0, Wt = 0, We = 0, Wd = 0, X = 0, OS = 0;
    int fails = 0, fallbacks = 0, learned = 0, iters = 0;
    signed char t = g.BCp[c];
    if (t != 30 && t != 31) {
        const double ie = prm.iselastic == 1 ? 1.0 / (prm.dt * f.mu_n[c]) : 1.0;
        const double exx = f.exxd[c], ezz = f.ezzd[c], exz = f.exz_n[c];
        const double sxx0 = f.sxxd0[c], szz0 = f.szzd0[c], sxz0 = f.sxz0_n[c];
        double E[6];
        eff_rates(exx, ezz, exz, sxx0, szz0, sxz0, ie, E);
        const double mu = f.mu_n[c], T = f.T[c], P = f.p[c], d0 = f.d0_n[c], phi0 = f.phi0_n[c];
        const double X0 = f.X0_n ? f.X0_n[c] : 0.0, P0 = f.p0_n ? f.p0_n[c] : 0.0;
        const double dil = f.dil_n[c], fric = f.fric_n[c], Coh = f.C_n[c], bet = f.bet_n[c];
        for (int p = 0; p < nph; p++) {
            double w = f.phase_perc_n[(size_t)p * nc + c];
            if (!(fabs(w) > 1.0e-13)) continue;
            visc_res o;
            float gs[2];
            if (guess) {
                const float2 q = guess[(size_t)p * nc + c];
                gs[0] = q.x; gs[1] = q.y;
            }
            visc_node_phase<FP32>(m, p, mu, ie, T, P, d0, phi0, X0, E, sxx0, szz0, sxz0, dil, fric, Coh, P0, bet, o,
                                  guess ? gs : nullptr);
            // labels may be the guess buffer itself: this thread read its entry above
            if (labels) labels[(size_t)p * nc + c] = make_float2(o.lab_x, o.lab_y);
            fails += o.ve_fail + o.vp_fail;
            fallbacks += o.fallback;
            iters += o.ve_its + o.vp_its;
            learned += o.learned;
            if (avg == 0) {
                eta += w * o.etaVE; eta_phys += w * o.eta; dexx += w * o.detadexx; dezz += w * o.detadezz;
                dgxz += w * o.detadexz / 2.0; dp += w * o.detadp;
            }
            if (avg == 0 || avg == 2) { sxx += w * o.txx; szz += w * o.tzz; sxz += w * o.txz; }
            VE += w * o.VEcoeff; eel += w * o.Eii_el; epl += w * o.Eii_pl; epwl += w * o.Eii_pwl;
            elin += w * o.Eii_lin; ecst += w * o.Eii_cst; dn += w * m.d.ph[p].igs_ref;
            eexp += w * o.Eii_exp; egbs += w * o.Eii_gbs;
            xel += w * o.Exx_el; xdi += w * o.Exx_diss; zel += w * o.Ezz_el; zdi += w * o.Ezz_diss;
            Wt += w * (o.txx * exx + o.tzz * ezz + (o.txx + o.tzz) * (exx + ezz) + 2.0 * o.txz * exz);
            Wd += w * (o.txx * o.Exx_diss + o.tzz * o.Ezz_diss + (o.txx + o.tzz) * (o.Exx_diss + o.Ezz_diss) +
                       2.0 * o.txz * o.Exz_diss);
            We += w * (o.txx * o.Exx_el + o.tzz * o.Ezz_el + (o.txx + o.tzz) * (o.Exx_el + o.Ezz_el) +
                       2.0 * o.txz * o.Exz_el);
            vxx += w * o.ddivpdexx; vzz += w * o.ddivpdezz; vxz += w * o.ddivpdexz / 2.0; vp += w * o.ddivpdp;
            pc += w * o.Pcorr; del += w * o.div_el; dpl += w * o.div_pl;
            X += w * o.X1; OS += w * o.OverS;
            if (avg == 1) {
                sxx += w * 1.0 / o.txx; szz += w * 1.0 / o.tzz; sxz += w * 1.0 / o.txz;
                eta += w * 1.0 / o.etaVE; eta_phys += w * 1.0 / o.eta;
                double ie2 = pow(o.etaVE, 2.0);
                dexx += w * o.detadexx / ie2; dezz += w * o.detadezz / ie2;
                dgxz += w * o.detadexz / 2.0 / ie2; dp += w * o.detadp / ie2;
            }
            if (avg == 2) {
                eta += w * log(o.etaVE); eta_phys += w * log(o.eta);
                dexx += w * o.detadexx / o.etaVE; dezz += w * o.detadezz / o.etaVE;
                dgxz += w * o.detadexz / 2.0 / o.etaVE; dp += w * o.detadp / o.etaVE;
            }
        }
        dn = 1.0 / dn;
        if (avg == 1) {
            sxx = 1.0 / sxx; szz = 1.0 / szz; sxz = 1.0 / sxz; eta = 1.0 / eta; eta_phys = 1.0 / eta_phys;
            double e2 = pow(eta, 2.0);
            dexx *= e2; dezz *= e2; dgxz *= e2; dp *= e2;
        }
        if (avg == 2) {
            eta = exp(eta); eta_phys = exp(eta_phys);
            dexx *= eta; dezz *= eta; dgxz *= eta; dp *= eta;
        }
    }
    put(f.eta_n, c, eta); put(f.eta_phys_n, c, eta_phys); put(f.VE_n, c, VE);
    put(f.sxxd, c, sxx); put(f.szzd, c, szz); put(f.sxz_n, c, sxz);
    put(f.eII_el, c, eel); put(f.eII_pl, c, epl); put(f.eII_pwl, c, epwl); put(f.eII_lin, c, elin);
    put(f.eII_cst, c, ecst); put(f.d_n, c, dn); put(f.eII_exp, c, eexp); put(f.eII_gbs, c, egbs);
    put(f.exx_el, c, xel); put(f.exx_diss, c, xdi); put(f.ezz_el, c, zel); put(f.ezz_diss, c, zdi);
    put(f.detadexx_n, c, dexx); put(f.detadezz_n, c, dezz); put(f.detadgxz_n, c, dgxz); put(f.detadp_n, c, dp);
    put(f.ddivpdexx_n, c, vxx); put(f.ddivpdezz_n, c, vzz); put(f.ddivpdgxz_n, c, vxz); put(f.ddivpdp_n, c, vp);
    put(f.p_corr, c, pc); put(f.div_u_el, c, del); put(f.div_u_pl, c, dpl); put(f.div_u_r, c, 0.0);
    put(f.Wtot, c, Wt); put(f.Wel, c, We); put(f.Wdiss, c, Wd); put(f.X_n, c, X); put(f.OverS_n, c, OS);
    count_local(counters, fails, fallbacks, learned, iters);
}

template <bool FP32>
__global__ void __launch_bounds__(128) k_viscosity_vertices(mdz_dgrid g, const __grid_constant__ visc_mats<FP32> m,
                                                             mdz_rheo_params prm,
                                                            mdz_fields f, int *__restrict__ counters,
                                                            const float2 *guess, float2 *labels) {
    int c = blockIdx.x * blockDim.x + threadIdx.x;
    int nv = g.Nx * g.Nz;
    if (c >= nv) return;
    const int avg = prm.eta_avg, nph = m.d.n_phases;
    double VE = 0, sxz = 0, eta_phys = 0, eta = 0, zel = 0, zdi = 0, dexx = 0, dezz = 0, dgxz = 0, dp = 0, X = 0,
           OS = 0;
    int fails = 0, fallbacks = 0, learned = 0, iters = 0;
    if (g.BCg[c] != 30) {
        const double ie = prm.iselastic == 1 ? 1.0 / (prm.dt * f.mu_s[c]) : 1.0;
        const double sxx0 = f.sxxd0_s[c], szz0 = f.szzd0_s[c], sxz0 = f.sxz0[c];
        double E[6];
        eff_rates(f.exxd_s[c], f.ezzd_s[c], f.exz[c], sxx0, szz0, sxz0, ie, E);
        const double mu = f.mu_s[c], T = f.T_s[c], P = f.P_s[c], d0 = f.d0_s[c], phi0 = f.phi0_s[c];
        const double X0 = f.X0_s ? f.X0_s[c] : 0.0, P0 = f.p0_s ? f.p0_s[c] : 0.0;
        const double dil = f.dil_s[c], fric = f.fric_s[c], Coh = f.C_s[c], bet = f.bet_s[c];
        for (int p = 0; p < nph; p++) {
            double w = f.phase_perc_s[(size_t)p * nv + c];
            if (!(fabs(w) > 1.0e-13)) continue;
            visc_res o;
            float gs[2];
            if (guess) {
                const float2 q = guess[(size_t)p * nv + c];
                gs[0] = q.x; gs[1] = q.y;
            }
            visc_node_phase<FP32>(m, p, mu, ie, T, P, d0, phi0, X0, E, sxx0, szz0, sxz0, dil, fric, Coh, P0, bet, o,
                                  guess ? gs : nullptr);
            // labels may be the guess buffer itself: this thread read its entry above
            if (labels) labels[(size_t)p * nv + c] = make_float2(o.lab_x, o.lab_y);
            fails += o.ve_fail + o.vp_fail;
            fallbacks += o.fallback;
            iters += o.ve_its + o.vp_its;
            learned += o.learned;
            if (avg == 0) {
                eta += w * o.etaVE; eta_phys += w * o.eta; dexx += w * o.detadexx; dezz += w * o.detadezz;
                dgxz += w * o.detadexz / 2.0; dp += w * o.detadp;
            }
            if (avg == 0 || avg == 2) sxz += w * o.txz;
            VE += w * o.VEcoeff; zel += w * o.Exz_el; zdi += w * o.Exz_diss; OS += w * o.OverS; X += w * o.X1;
            if (avg == 1) {
                sxz += w * 1.0 / o.txz; eta += w * 1.0 / o.etaVE; eta_phys += w * 1.0 / o.eta;
                double ie2 = pow(o.etaVE, 2.0);
                dexx += w * o.detadexx / ie2; dezz += w * o.detadezz / ie2;
                dgxz += w * o.detadexz / 2.0 / ie2; dp += w * o.detadp / ie2;
            }
            if (avg == 2) {
                eta += w * log(o.etaVE); eta_phys += w * log(o.eta);
                dexx += w * o.detadexx / o.etaVE; dezz += w * o.detadezz / o.etaVE;
                dgxz += w * o.detadexz / 2.0 / o.etaVE; dp += w * o.detadp / o.etaVE;
            }
        }
        if (avg == 1) {
            sxz = 1.0 / sxz; eta = 1.0 / eta; eta_phys = 1.0 / eta_phys;
            double e2 = pow(eta, 2.0);
            dexx *= e2; dezz *= e2; dgxz *= e2; dp *= e2;
        }
        if (avg == 2) {
            eta = exp(eta); eta_phys = exp(eta_phys);
            dexx *= eta; dezz *= eta; dgxz *= eta; dp *= eta;
        }
    }
    put(f.VE_s, c, VE); put(f.sxz, c, sxz); put(f.eta_phys_s, c, eta_phys); put(f.eta_s, c, eta);
    put(f.exz_el, c, zel); put(f.exz_diss, c, zdi);
    put(f.detadexx_s, c, dexx); put(f.detadezz_s, c, dezz); put(f.detadgxz_s, c, dgxz); put(f.detadp_s, c, dp);
    put(f.X_s, c, X); put(f.OverS_s, c, OS);
    count_local(counters, fails, fallbacks, learned, iters);
}

// ---------------------------------------------------------------------------
// Rheological operators (isotropic): Picard D = 2 eta I / eta; Newton adds the
// tangent terms 2 deta/dE * G.
__global__ void k_operators(mdz_dgrid g, mdz_rheo_params prm, mdz_fields f, int jacobian) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    int nc = g.ncx * g.ncz, nv = g.Nx * g.Nz;
    if (i < nc) {
        int k = i;
        double d11 = 0, d12 = 0, d13 = 0, d14 = 0, d21 = 0, d22 = 0, d23 = 0, d24 = 0;
        if (g.BCp[k] != 30 && g.BCp[k] != 31) {
            double eta = f.eta_n[k];
            d11 = 2.0 * eta; d22 = 2.0 * eta;
            if (jacobian) {
                double ie = prm.iselastic == 1 ? 1.0 / (prm.dt * f.mu_n[k]) : 1.0, E[6];
                eff_rates(f.exxd[k], f.ezzd[k], f.exz_n[k], f.sxxd0[k], f.szzd0[k], f.sxz0_n[k], ie, E);
                // K = 0 (incompressible): the K*dt*ddivp terms vanish
                d11 += 2.0 * f.detadexx_n[k] * E[3];
                d12 = 2.0 * f.detadezz_n[k] * E[3];
                d13 = 2.0 * f.detadgxz_n[k] * E[3];
                d14 = 2.0 * f.detadp_n[k] * E[0];
                d21 = 2.0 * f.detadexx_n[k] * E[4];
                d22 += 2.0 * f.detadezz_n[k] * E[4];
                d23 = 2.0 * f.detadgxz_n[k] * E[4];
                d24 = 2.0 * f.detadp_n[k] * E[1];
            }
        }
        f.D11_n[k] = d11; f.D12_n[k] = d12; f.D13_n[k] = d13; f.D14_n[k] = d14;
        f.D21_n[k] = d21; f.D22_n[k] = d22; f.D23_n[k] = d23; f.D24_n[k] = d24;
    }
    if (i < nv) {
        int k = i;
        double d31 = 0, d32 = 0, d33 = 0, d34 = 0;
        if (g.BCg[k] != 30) {
            double eta = f.eta_s[k];
            d33 = eta;
            if (jacobian) {
                double ie = prm.iselastic == 1 ? 1.0 / (prm.dt * f.mu_s[k]) : 1.0, E[6];
                eff_rates(f.exxd_s[k], f.ezzd_s[k], f.exz[k], f.sxxd0_s[k], f.szzd0_s[k], f.sxz0[k], ie, E);
                d31 = 2.0 * f.detadexx_s[k] * E[5];
                d32 = 2.0 * f.detadezz_s[k] * E[5];
                d33 += 2.0 * f.detadgxz_s[k] * E[5];
                d34 = 2.0 * f.detadp_s[k] * E[2];
            }
        }
        f.D31_s[k] = d31; f.D32_s[k] = d32; f.D33_s[k] = d33; f.D34_s[k] = d34;
    }
}

// ---------------------------------------------------------------------------
// Momentum RHS (body force + elastic stress history), continuity RHS = 0.
// A CTA takes a 32 x 8 tile of the index box; the visco-elastic factors
// eta / (mu dt) times the old stresses, which four rows each read, are formed
// once per centroid and vertex of the tile and its southern and western ring in
// shared memory: eight FP64 divisions per node before, two now, the same
// products.  1024 x 512 cells: 99 -> 50 us.
constexpr int RHS_W = 32, RHS_H = 8;

__global__ void __launch_bounds__(RHS_W *RHS_H) k_rhs(mdz_dgrid g, mdz_rheo_params prm, double gx, double gz, mdz_fields f) {
    // centroids (i0 - 1 .., j0 - 1 ..): eta / (mu dt) sxxd0, szzd0; vertices (i0 - 1 .., j0 - 1 ..): sxz0
    __shared__ double qx[RHS_H + 1][RHS_W + 1], qz[RHS_H + 1][RHS_W + 1], qs[RHS_H + 1][RHS_W + 1];
    const int Nx = g.Nx, Nz = g.Nz, ncx = g.ncx, ncz = g.ncz;
    const int tx = threadIdx.x % RHS_W, ty = threadIdx.x / RHS_W, i0 = blockIdx.x * RHS_W, j0 = blockIdx.y * RHS_H;
    const double dt = prm.dt;
    const bool elastic = prm.iselastic == 1;
    if (elastic) {
        for (int t = threadIdx.x; t < (RHS_W + 1) * (RHS_H + 1); t += RHS_W * RHS_H) {
            const int a = t % (RHS_W + 1), b = t / (RHS_W + 1), k = i0 - 1 + a, l = j0 - 1 + b;
            double vx = 0.0, vz = 0.0, vs = 0.0;
            if (k >= 0 && l >= 0 && k < ncx && l < ncz && g.BCp[k + l * ncx] == -1) {
                const int c = k + l * ncx;
                const double h = f.eta_n[c] / (f.mu_n[c] * dt);
                vx = h * f.sxxd0[c];
                vz = h * f.szzd0[c];
            }
            if (k >= 0 && l >= 0 && k < Nx && l < Nz && g.BCg[k + l * Nx] != 30) {
                const int c = k + l * Nx;
                vs = f.eta_s[c] / (f.mu_s[c] * dt) * f.sxz0[c];
            }
            qx[b][a] = vx; qz[b][a] = vz; qs[b][a] = vs;
        }
        __syncthreads();
    }
    const int k = i0 + tx, l = j0 + ty;
    if (k < Nx && l <= Nz) {   // Vx (k, l): centroids (k - 1, l - 1), (k, l - 1), vertices (k, l - 1), (k, l)
        const int c = k + l * Nx;
        double r = 0.0;
        if (f.gx) f.gx[c] = gx;
        const signed char t = g.BCu[c];
        if (l > 0 && l < Nz && (t == -1 || t == 2 || t == -2)) {
            r = -gx * (0.5 * (f.rho_s[c - Nx] + f.rho_s[c]));
            if (elastic && k > 0 && k < Nx - 1) {
                const int p = k + (l - 1) * ncx;
                if (g.BCp[p] == -1) r -= g.idx * qx[ty][tx + 1];
                if (g.BCp[p - 1] == -1) r -= g.idx * -qx[ty][tx];
                if (g.BCg[c] != 30 && g.BCu[c + Nx] != 13) r -= g.idz * qs[ty + 1][tx + 1];
                if (g.BCg[c - Nx] != 30 && g.BCu[c - Nx] != 13) r -= g.idz * -qs[ty][tx + 1];
            }
        }
        f.roger_x[c] = -r;
    }
    if (k <= Nx && l < Nz) {   // Vz (k, l): centroids (k - 1, l - 1), (k - 1, l), vertices (k - 1, l), (k, l)
        const int c = k + l * (Nx + 1);
        double r = 0.0;
        if (f.gz) f.gz[c] = gz;
        if (k > 0 && k < Nx && g.BCv[c] == -1) {
            const int p = k - 1 + (l - 1) * ncx, q = k + l * Nx;
            r = -gz * (0.5 * ((l > 0 ? f.rho_n[p] : 0.0) + (l < Nz - 1 ? f.rho_n[p + ncx] : 0.0)));
            if (elastic && l > 0 && l < Nz - 1) {
                if (g.BCp[p + ncx] == -1) r -= g.idz * qz[ty + 1][tx];
                if (g.BCp[p] == -1) r -= g.idz * -qz[ty][tx];
                if (g.BCg[q] != 30 && g.BCv[c + 1] != 13) r -= g.idx * qs[ty + 1][tx + 1];
                if (g.BCg[q - 1] != 30 && g.BCv[c - 1] != 13) r -= g.idx * -qs[ty + 1][tx];
            }
        }
        f.roger_z[c] = -r;
    }
    if (k < ncx && l < ncz) {
        const int c = k + l * ncx;
        if (g.BCp[c] != 30 && g.BCp[c] != 31) f.rhs_p[c] = 0.0;
    }
}

// ---------------------------------------------------------------------------
// Device-level launchers (used by the host drop-ins and by the time step).
mdz_status mdz_dev_strain_rates(mdz_ctx *ctx, const mdz_fields &f, cudaStream_t st) {
    const mdz_dgrid &g = ctx->g;
    const int nv = g.Nx * g.Nz;   // (more than the centroids)
    k_strain<<<mdz_blocks(nv), MDZ_THREADS, 0, st>>>(g, f.u, f.v, f.div_u, f.exxd, f.ezzd, f.exz);
    MDZ_LAUNCHED(ctx);
    k_strain_averages<<<mdz_blocks(nv), MDZ_THREADS, 0, st>>>(g, f.exz, f.exz_n,
                                                              c2v_fields<2>{{f.exxd, f.ezzd}, {f.exxd_s, f.ezzd_s}});
    MDZ_LAUNCHED(ctx);
    return MDZ_OK;
}

mdz_status mdz_dev_c2v(mdz_ctx *ctx, const double *cen, double *ver, cudaStream_t st) {
    k_c2v<1><<<mdz_blocks(ctx->g.Nx * ctx->g.Nz), MDZ_THREADS, 0, st>>>(ctx->g, c2v_fields<1>{{cen}, {ver}});
    MDZ_LAUNCHED(ctx);
    return MDZ_OK;
}

mdz_status mdz_dev_v2c(mdz_ctx *ctx, double *cen, const double *ver, cudaStream_t st) {
    k_v2c<<<mdz_blocks(ctx->g.ncx * ctx->g.ncz), MDZ_THREADS, 0, st>>>(ctx->g, cen, ver);
    MDZ_LAUNCHED(ctx);
    return MDZ_OK;
}

mdz_status mdz_check_materials(mdz_ctx *ctx, const mdz_materials *m) {
    if (m->n_phases < 1 || m->n_phases > MDZ_MAX_PHASES || m->n_phases > ctx->n_phases)
        return mdz_fail(ctx, MDZ_ERR_ARG, "materials: %d phases (context has %d)", m->n_phases, ctx->n_phases);
    for (int p = 0; p < m->n_phases; p++) {
        if (m->gs[p] || m->reac_soft[p] || m->phase_mix[p])
            return mdz_fail(ctx, MDZ_ERR_UNSUPPORTED,
                            "phase %d: grain-size evolution and reaction mixing are not implemented", p);
        if (m->gbsv[p] && m->ngbs[p] <= 0) return mdz_fail(ctx, MDZ_ERR_ARG, "phase %d: ngbs must be > 0", p);
        if (m->expv[p] && !(m->Gexp[p] > 0 && m->Gexp[p] < 1 && m->Eexp[p] > 0 && m->Sexp[p] > 0))
            return mdz_fail(ctx, MDZ_ERR_ARG, "phase %d: Peierls creep needs 0 < Gexp < 1, Eexp > 0, Sexp > 0", p);
        if (m->pwlv[p] && m->npwl[p] <= 0) return mdz_fail(ctx, MDZ_ERR_ARG, "phase %d: npwl must be > 0", p);
        if (m->linv[p] && m->nlin[p] <= 0) return mdz_fail(ctx, MDZ_ERR_ARG, "phase %d: nlin must be > 0", p);
        if (m->n_vp[p] <= 0) return mdz_fail(ctx, MDZ_ERR_ARG, "phase %d: n_vp must be > 0", p);
    }
    return MDZ_OK;
}

// ---------------------------------------------------------------------------
// Learned guess: per (node, phase) MLP inference, one warp per 32 nodes and a
// warp-synchronous tensor-core pass per phase present in the warp.
__device__ __forceinline__ double eii_of(const double *E, const mdz_rheo_params &prm) {
    const double Eyy = -(E[0] + E[1]);
    double Eii = sqrt(0.5 * (E[0] * E[0] + E[1] * E[1] + Eyy * Eyy) + E[2] * E[2]);
    if (Eii * prm.scale_E < 1e-30) Eii = 1e-30 / prm.scale_E;
    return Eii;
}

template <bool CENT>
__global__ void __launch_bounds__(256) k_mlp_guess(mdz_dgrid g, int nph, mdz_rheo_params prm, mdz_fields f,
                                                   mdz_mlp_norm nm, const unsigned char *__restrict__ packed,
                                                   float2 *__restrict__ guess) {
    extern __shared__ __align__(16) unsigned char sm[];
    __nv_bfloat16 *XS = reinterpret_cast<__nv_bfloat16 *>(sm + MLP_PACK_BYTES);
    float *YS = reinterpret_cast<float *>(XS + 8 * 32 * MLP_S1);
    mlp_load_weights(sm, packed);
    for (int i = threadIdx.x; i < 8 * 32 * MLP_S1; i += blockDim.x) XS[i] = __float2bfloat16_rn(0.f);
    __syncthreads();
    const mlp_w W = mlp_views(sm);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    __nv_bfloat16 *xs = XS + warp * 32 * MLP_S1;
    float *ys = YS + warp * 64;
    const int nn = CENT ? g.ncx * g.ncz : g.Nx * g.Nz;
    for (int base = (blockIdx.x * 8 + warp) * 32; base < nn; base += gridDim.x * 8 * 32) {
        const int c = base + lane;
        bool act = c < nn;
        if (act) act = CENT ? (g.BCp[c] != 30 && g.BCp[c] != 31) : (g.BCg[c] != 30);
        double Eii = 1.0 / prm.scale_E, T = ZEROC / prm.scale_T, P = 0.0;
        if (act) {
            double E[6];
            if (CENT) {
                const double ie = prm.iselastic == 1 ? 1.0 / (prm.dt * f.mu_n[c]) : 1.0;
                eff_rates(f.exxd[c], f.ezzd[c], f.exz_n[c], f.sxxd0[c], f.szzd0[c], f.sxz0_n[c], ie, E);
                T = f.T[c];
                P = f.p[c];
            } else {
                const double ie = prm.iselastic == 1 ? 1.0 / (prm.dt * f.mu_s[c]) : 1.0;
                eff_rates(f.exxd_s[c], f.ezzd_s[c], f.exz[c], f.sxxd0_s[c], f.szzd0_s[c], f.sxz0[c], ie, E);
                T = f.T_s[c];
                P = f.P_s[c];
            }
            Eii = eii_of(E, prm);
            if (T < ZEROC / prm.scale_T) T = ZEROC / prm.scale_T;
        }
        for (int p = 0; p < nph; p++) {
            const double w = act ? (CENT ? f.phase_perc_n[(size_t)p * nn + c] : f.phase_perc_s[(size_t)p * nn + c]) : 0.0;
            const bool need = act && fabs(w) > 1.0e-13;
            if (!__any_sync(0xffffffffu, need)) continue;
            float x[8];
            mlp_inputs(nm, prm, Eii, T, P, prm.dt, p, x);
            *reinterpret_cast<uint4 *>(xs + lane * MLP_S1) =
                make_uint4(mlp_pack2(x[0], x[1]), mlp_pack2(x[2], x[3]), mlp_pack2(x[4], x[5]), mlp_pack2(x[6], x[7]));
            __syncwarp();
            mlp_warp_infer(W, xs, ys);
            __syncwarp();
            if (need) guess[(size_t)p * nn + c] = make_float2(ys[2 * lane], ys[2 * lane + 1]);
            __syncwarp();
        }
    }
}

mdz_status mdz_dev_mlp_guess(mdz_ctx *ctx, const mdz_materials *m, const mdz_rheo_params *prm, const mdz_fields &f,
                             float2 *guess_n, float2 *guess_s, cudaStream_t st) {
    const mdz_dgrid &g = ctx->g;
    const int nc = g.ncx * g.ncz, nv = g.Nx * g.Nz;
    const size_t smem = MLP_PACK_BYTES + 8 * 32 * MLP_S1 * 2 + 8 * 64 * 4;
    int dev = 0, sms = 152;
    cudaGetDevice(&dev);
    cudaDeviceGetAttribute(&sms, cudaDevAttrMultiProcessorCount, dev);
    auto grid = [&](int n) { int b = (n + 255) / 256; return b < 4 * sms ? (b < 1 ? 1 : b) : 4 * sms; };
    cudaEvent_t ev;
    mdz_prof_begin(ctx, MDZ_PROF_MLP, st, &ev);
    k_mlp_guess<true><<<grid(nc), 256, smem, st>>>(g, m->n_phases, *prm, f, ctx->mlp->norm, ctx->mlp->packed, guess_n);
    MDZ_LAUNCHED(ctx);
    k_mlp_guess<false><<<grid(nv), 256, smem, st>>>(g, m->n_phases, *prm, f, ctx->mlp->norm, ctx->mlp->packed, guess_s);
    MDZ_LAUNCHED(ctx);
    // per node: 6 FP64 rate/stress inputs, mu, T, P, the phase fractions, the tag; one float2 per phase out
    const double bytes = (double)(nc + nv) * (8.0 * (9 + m->n_phases) + 1 + 8.0 * m->n_phases);
    mdz_prof_end(ctx, MDZ_PROF_MLP, bytes, st, ev);
    return MDZ_OK;
}

// Training tuples: (strain rate, T, P, dt, phase) drawn from the ranges with a
// counter-based generator, labelled by the plain local solve.
__device__ __forceinline__ double mlp_u01(unsigned long long seed, long long i, int k) {
    unsigned long long z = seed + 0x9E3779B97F4A7C15ull * (unsigned long long)(5 * i + k + 1);
    z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
    z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
    z ^= z >> 31;
    return (double)(z >> 11) * (1.0 / 9007199254740992.0);
}

__global__ void __launch_bounds__(128) k_mlp_samples(long long n, unsigned long long seed, mdz_materials m,
                                                     const __grid_constant__ visc_mats<false> mk,
                                                     mdz_rheo_params prm, double lo0, double hi0, double lo1,
                                                     double hi1, double lo2, double hi2, double lo3, double hi3,
                                                     mdz_mlp_norm nm, uint4 *__restrict__ X, float2 *__restrict__ Y) {
    const long long i = (long long)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const double Eii = pow(10.0, lo0 + (hi0 - lo0) * mlp_u01(seed, i, 0)) / prm.scale_E;
    double T = (lo1 + (hi1 - lo1) * mlp_u01(seed, i, 1)) / prm.scale_T;
    const double P = (lo2 + (hi2 - lo2) * mlp_u01(seed, i, 2)) / prm.scale_S;
    const double dt = pow(10.0, lo3 + (hi3 - lo3) * mlp_u01(seed, i, 3)) * prm.scale_E;
    int ph = (int)(mlp_u01(seed, i, 4) * m.n_phases);
    if (ph > m.n_phases - 1) ph = m.n_phases - 1;
    mdz_rheo_params q = prm;
    q.dt = dt;
    if (T < ZEROC / q.scale_T) T = ZEROC / q.scale_T;
    visc_res o;
    visc_prm<double> vq = mk.d.prm;   // the tuple's own time step
    vq.dt = dt;
    vq.idt = 1.0 / dt;
    visc_local_t<double>(mk.d.ph[ph], vq, m.mu[ph], 1.0 / (dt * m.mu[ph]), T, P, m.gs_ref[ph], 0.0, 0.0, Eii, -Eii, 0.0,
                         0.0, 0.0, 0.0, m.psi[ph], m.phi[ph], m.C[ph], P, m.bet[ph], o, nullptr);
    float2 lab = mlp_labels(o.eta_ve, o.eta_up, o.gdot, Eii);
    lab.x = fminf(fmaxf(lab.x, -8.f), 1.f);
    lab.y = fminf(fmaxf(lab.y, 0.f), 1.f);
    float x[8];
    mlp_inputs(nm, q, Eii, T, P, dt, ph, x);
    X[i] = make_uint4(mlp_pack2(x[0], x[1]), mlp_pack2(x[2], x[3]), mlp_pack2(x[4], x[5]), mlp_pack2(x[6], x[7]));
    Y[i] = lab;
}

mdz_status mdz_dev_mlp_samples(mdz_ctx *ctx, const mdz_materials *m, const mdz_rheo_params *prm, long long n,
                               unsigned long long seed, const double lo[4], const double hi[4],
                               const mdz_mlp_norm &norm, uint4 *X, float2 *Y, cudaStream_t st) {
    k_mlp_samples<<<(unsigned)((n + 127) / 128), 128, 0, st>>>(n, seed, *m, visc_mats<false>{make_visc_mat<double>(*m, *prm)}, *prm, lo[0], hi[0], lo[1], hi[1], lo[2],
                                                                hi[2], lo[3], hi[3], norm, X, Y);
    MDZ_LAUNCHED(ctx);
    return MDZ_OK;
}

mdz_status mdz_dev_viscosity(mdz_ctx *ctx, const mdz_materials *m, const mdz_rheo_params *prm, const mdz_fields &f,
                             int *d_counters, cudaStream_t st, bool learned, bool fp32, int warm) {
    const mdz_dgrid &g = ctx->g;
    int nc = g.ncx * g.ncz, nv = g.Nx * g.Nz;
    // vertex copies of centroid fields (NonNewtonianViscosityGrid :979-983)
    mdz_status s;
    k_c2v<5><<<mdz_blocks(nv), MDZ_THREADS, 0, st>>>(g, c2v_fields<5>{{f.div_u, f.T, f.p, f.d0_n, f.phi0_n},
                                                                      {f.div_u_s, f.T_s, f.P_s, f.d0_s, f.phi0_s}});
    MDZ_LAUNCHED(ctx);
    const float2 *guess_n = nullptr, *guess_s = nullptr;
    float2 *lab_n = nullptr, *lab_s = nullptr;
    if (learned && !fp32) {
        float2 *buf = mdz_mlp_guess_buffer(ctx, (size_t)m->n_phases * (nc + nv));
        if (!buf) return mdz_fail(ctx, MDZ_ERR_CUDA, "learned guess: buffer allocation failed");
        if (warm != 2)
            if ((s = mdz_dev_mlp_guess(ctx, m, prm, f, buf, buf + (size_t)m->n_phases * nc, st)) != MDZ_OK) return s;
        guess_n = buf;
        guess_s = buf + (size_t)m->n_phases * nc;
        if (warm >= 1) { lab_n = buf; lab_s = buf + (size_t)m->n_phases * nc; }
    }
    cudaEvent_t ev;
    mdz_prof_begin(ctx, MDZ_PROF_VISCOSITY, st, &ev);
    if (fp32) {
        const visc_mats<true> mk{make_visc_mat<double>(*m, *prm), make_visc_mat<float>(*m, *prm)};
        k_viscosity_centroids<true><<<mdz_blocks(nc, 128), 128, 0, st>>>(g, mk, *prm, f, d_counters, guess_n, lab_n);
        MDZ_LAUNCHED(ctx);
        k_viscosity_vertices<true><<<mdz_blocks(nv, 128), 128, 0, st>>>(g, mk, *prm, f, d_counters, guess_s, lab_s);
    } else {
        const visc_mats<false> mk{make_visc_mat<double>(*m, *prm)};
        k_viscosity_centroids<false><<<mdz_blocks(nc, 128), 128, 0, st>>>(g, mk, *prm, f, d_counters, guess_n, lab_n);
        MDZ_LAUNCHED(ctx);
        k_viscosity_vertices<false><<<mdz_blocks(nv, 128), 128, 0, st>>>(g, mk, *prm, f, d_counters, guess_s, lab_s);
    }
    MDZ_LAUNCHED(ctx);
    // algorithmic bytes: per centroid 17 + n_phases FP64 inputs and 35 outputs,
    // per vertex 17 + n_phases inputs and 12 outputs, plus the tags
    double bytes = (double)nc * (8.0 * (17 + m->n_phases + 35) + 1) + (double)nv * (8.0 * (17 + m->n_phases + 12) + 1);
    mdz_prof_end(ctx, MDZ_PROF_VISCOSITY, bytes, st, ev);
    return MDZ_OK;
}

mdz_status mdz_dev_operators(mdz_ctx *ctx, const mdz_rheo_params *prm, const mdz_fields &f, int jacobian,
                             cudaStream_t st) {
    const mdz_dgrid &g = ctx->g;
    int n = g.Nx * g.Nz;
    k_operators<<<mdz_blocks(n), MDZ_THREADS, 0, st>>>(g, *prm, f, jacobian);
    MDZ_LAUNCHED(ctx);
    return MDZ_OK;
}

mdz_status mdz_dev_rhs(mdz_ctx *ctx, const mdz_rheo_params *prm, double gx, double gz, const mdz_fields &f,
                       cudaStream_t st) {
    const mdz_dgrid &g = ctx->g;
    k_rhs<<<dim3((g.Nx + RHS_W) / RHS_W, (g.Nz + RHS_H) / RHS_H), RHS_W * RHS_H, 0, st>>>(g, *prm, gx, gz, f);
    MDZ_LAUNCHED(ctx);
    return MDZ_OK;
}
