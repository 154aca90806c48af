// fsg_mag.cu -- magnetic path: MagLineopCalc (Zeeman-split Faraday-Voigt opacity into the six
// profiles) and MagRadTranCalc (Stokes DELO-Bezier solver, plane-parallel and spherical).  Built -fmad=false:
// FP64 throughout, in the reference's operation order.
//
//   k_mag_center    MagLineopCalc central pass (synth.f90:1182-1275), one warp per line: Zeeman shifts scaled to
//                   FP32 (Kz |B| lambda^2, synth.f90:1193-1194), centre test (LineOpacity2),
//                   doubling search with MagLineOpacity2 and RefineIdx bisection
//                   (opacity.f90:468-520, 611-675)
//   (the sums, MagLineOpacity1/3, are in fsg_accum64.cu and fsg_magfast.cu)
//   k_stokes_thr    StokesPrfPP (solver.f90:265-394) + Solve4x4 (solver.f90:541-588), one thread per
//                   (wavelength, angle); k_stokes_flux the Stokes-I flux quadrature
//   k_stokes_sph    StokesPrfSph (solver.f90:402-538) along the rays of a spherical model, one thread per
//                   (wavelength, ray)
#include "fsg_fp64.cuh"

#include <algorithm>
#include <math.h>
#include <string.h>
#include <vector>

// MagLineOpacity2 at one wavelength, max over depths of LineOpac/ContOpacL (opacity.f90:468-520)
// over the depths t0, t0 + tstep, ... (a lane's share when a warp takes the line)
__device__ double mag_lineop2_max(const AtmView &A, const XCoef &XC, double Wl, double wlc, int ihe,
                                  const ZView &Z, int64_t i, int iwl, double dW, const float *vtab,
                                  const double *anode, const double *aida, int t0 = 0, int tstep = 1) {
    const int nt = A.ntau;
    double mx = -1.0e308;
    const int np = Z.npi[i], ns = Z.nsi[i];
    const float *spi = Z.splpi + Z.pi_off[i], *ssi = Z.splsi + Z.si_off[i];
    const float *rpi = Z.strpi + Z.pi_off[i], *rsi = Z.strsi + Z.si_off[i];
    double dWl0 = Wl - wlc;
    for (int t = t0; t < nt; t += tstep) {
        double cop, vv, av;
        xline_depth(A, t, XC, &cop, &vv, &av);
        double dWl = dWl0;
        if (ihe > 0) dWl = dWl0 - A.heshf[(ihe - 1) * nt + t];
        VLine64 VL = vline64(anode, aida, av);
        double Pp = 0.0, Ps = 0.0;
        for (int k = 0; k < np; k++) Pp = Pp + (double)rpi[k] * hvoigt_line64(vtab, VL, (dWl - (double)spi[k]) * vv);
        for (int k = 0; k < ns; k++) Ps = Ps + (double)rsi[k] * hvoigt_line64(vtab, VL, (dWl - (double)ssi[k]) * vv);
        double lo = fmax(0.5 * Ps, 0.5 * Pp + 0.25 * Ps) * cop;
        if (A.motype == 1) lo = lo / A.contstd[t];
        mx = fmax(mx, lo / cont_center(A, iwl, dW, t));
    }
    return mx;
}

__device__ __forceinline__ double warp_max(double v) {
    for (int o = 16; o > 0; o >>= 1) v = fmax(v, __shfl_xor_sync(0xffffffffu, v, o));
    return v;
}

// MagLineOpacity2's maximum over depths (opacity.f90:468-520), the lanes of a warp over the depths
__device__ __forceinline__ double mag_lineop2_max_warp(const AtmView &A, const XCoef &XC, double Wl, double wlc,
                                                       int ihe, const ZView &Z, int64_t i, int iwl, double dW,
                                                       const float *vtab, const double *anode, const double *aida,
                                                       int lane) {
    return warp_max(mag_lineop2_max(A, XC, Wl, wlc, ihe, Z, i, iwl, dW, vtab, anode, aida, lane, 32));
}

// Magnetic central pass, one warp per line: the lanes share the depth loops of the centre test and of
// every MagLineOpacity2 evaluation of the window search (maxima over depths, so the lanes' partial
// maxima combine exactly), the search itself is warp-uniform.
__global__ void k_mag_center(AtmView A, LineView L, ZView Z, double Bsplit, const float *__restrict__ vtab,
                             const double *__restrict__ anode, const double *__restrict__ aida,
                             int32_t *flags, int32_t *ileft, int32_t *iright, unsigned long long *nkeep) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= L.n) return;                                // whole warps leave together
    const int nt = A.ntau;
    int f = 0;
    if (L.ismol && L.ismol[i]) f |= FSG_F_MOL;
    if (L.gvdw[i] > 10.0f) f |= FSG_F_ABO;
    double wlc = L.wl[i] - A.wfirst;
    double w = wlc + A.wfirst;
    // scale the pattern by Kz |B| lambda^2, rounded to FP32 (synth.f90:1193-1194)
    const int np = Z.npi[i], ns = Z.nsi[i];
    double smx_pi = -3.4028234663852886e38, smx_si = -3.4028234663852886e38;
    for (int k = lane; k < np; k += 32) {
        float v = (float)((double)Z.rawpi[Z.pi_off[i] + k] * Bsplit * (w * w));
        Z.splpi[Z.pi_off[i] + k] = v;
        smx_pi = fmax(smx_pi, fabs((double)v));
    }
    for (int k = lane; k < ns; k += 32) {
        float v = (float)((double)Z.rawsi[Z.si_off[i] + k] * Bsplit * (w * w));
        Z.splsi[Z.si_off[i] + k] = v;
        smx_si = fmax(smx_si, fabs((double)v));
    }
    const double SplMax = fmax(warp_max(smx_si), warp_max(smx_pi));
    __syncwarp();                                        // every lane's scaled shifts are visible below
    XCoef XC;
    xline_setup(A, L, i, wlc, f, &XC);
    if (XC.IxHe > 0) f |= (XC.IxHe << 8);
    int ihe = XC.IxHe;
    int iwl = waveidx(A, wlc);
    double dW = (wlc - A.wave[iwl - 1]) / (A.wave[iwl] - A.wave[iwl - 1]);
    // non-magnetic centre opacity (synth.f90:1215-1224)
    double mx = -1.0e308;
    for (int t = lane; t < nt; t += 32) {
        double cop, vv, av;
        xline_depth(A, t, XC, &cop, &vv, &av);
        double dWl = 0.0;
        if (ihe > 0) dWl = 0.0 - A.heshf[(ihe - 1) * nt + t];
        double lo = hvoigt64(vtab, anode, aida, av, dWl * vv) * cop;
        if (A.motype == 1) lo = lo / A.contstd[t];
        mx = fmax(mx, lo / cont_center(A, iwl, dW, t));
    }
    mx = warp_max(mx);
    int il = 1, ir = A.nwl;
    if (mx < A.epsopac) f |= FSG_F_WEAK;
    else {
        // doubling search (synth.f90:1233-1272)
        for (int idw = 0; idw < 64; idw++) {
            double dWo = (0.2 * ldexp(1.0, idw)) * (wlc + A.wfirst) / 5e3;
            double Wl = wlc + SplMax + dWo;
            double m2 = mag_lineop2_max_warp(A, XC, Wl, wlc, ihe, Z, i, iwl, dW, vtab, anode, aida, lane);
            if (m2 < A.epsopac) {
                // RefineIdx (opacity.f90:611-675), magnetic branch
                int isw, ikw;
                if (wlc > 0.5 * (A.wave[0] + A.wave[A.nwl - 1])) { isw = -1; ikw = 0; }
                else { isw = 1; ikw = 1; }
                int ia, ib;
                if (idw == 0) ia = waveidx(A, wlc + (double)isw * SplMax) + ikw;
                else {
                    double d1 = (0.2 * ldexp(1.0, idw - 1)) * (wlc + A.wfirst) / 5e3;
                    ia = waveidx(A, wlc + (double)isw * (SplMax + d1)) + ikw;
                }
                ib = waveidx(A, wlc + (double)isw * (SplMax + dWo)) + ikw;
                for (int it = 0; it < 64 && abs(ia - ib) > 1; it++) {
                    int im = (ia + ib) / 2;
                    double m3 = mag_lineop2_max_warp(A, XC, A.wave[im - 1], wlc, ihe, Z, i, iwl, dW, vtab, anode,
                                                     aida, lane);
                    if (m3 < A.epsopac) ib = im; else ia = im;
                }
                if (isw == 1) { ir = ia; il = waveidx(A, 2.0 * wlc - A.wave[ia - 1]); }
                else { il = ia; ir = waveidx(A, 2.0 * wlc - A.wave[ia - 1]) + 1; }
                break;
            } else if (wlc - SplMax - dWo < A.wave[0] && wlc + SplMax + dWo > A.wave[A.nwl - 1]) break;
        }
    }
    if (lane == 0) {
        flags[i] = f; ileft[i] = il; iright[i] = ir;
        if (!(f & FSG_F_WEAK)) atomicAdd(nkeep, 1ull);
    }
}

// six profiles of one line at one wavelength for depth t (MagLineOpacity1/3 inner loops)
__device__ __forceinline__ void mag_profiles_t(const AtmView &A, int t, double Wl, double wlc, int ihe,
                                               const ZView &Z, int64_t i, double cop, double vv, double av,
                                               const float2 *fvtab, const double *anode, const double *aida,
                                               double *m) {
    VLine64 FL = vline64(anode, aida, av);
    double Xn = cop, sc = vv, Vbase = (Wl - wlc) * sc;
    if (ihe > 0) Vbase = Vbase - A.heshf[(ihe - 1) * A.ntau + t] * sc;
    const int np = Z.npi[i], ns = Z.nsi[i];
    const float *spi = Z.splpi + Z.pi_off[i], *ssi = Z.splsi + Z.si_off[i];
    const float *rpi = Z.strpi + Z.pi_off[i], *rsi = Z.strsi + Z.si_off[i];
    for (int k = 0; k < np; k++) {
        double V = Vbase - (double)spi[k] * sc, Vg, Fv;
        fvoigt_line64(fvtab, FL, V, &Vg, &Fv);
        double Str = Xn * (double)rpi[k];
        m[0] = m[0] + Str * Vg; m[3] = m[3] + Str * Fv;
    }
    int Nsh = ns / 2;
    for (int k = 0; k < Nsh; k++) {
        double V = Vbase - (double)ssi[k] * sc, Vg, Fv;
        fvoigt_line64(fvtab, FL, V, &Vg, &Fv);
        double Str = Xn * (double)rsi[k];
        m[1] = m[1] + Str * Vg; m[4] = m[4] + Str * Fv;
    }
    for (int k = Nsh; k < ns; k++) {
        double V = Vbase - (double)ssi[k] * sc, Vg, Fv;
        fvoigt_line64(fvtab, FL, V, &Vg, &Fv);
        double Str = Xn * (double)rsi[k];
        m[2] = m[2] + Str * Vg; m[5] = m[5] + Str * Fv;
    }
}

// ================================================================================================
// Stokes solvers (solver.f90:265-538).  The per-depth propagation data are the 6 distinct elements of
// the normalised 4x4 matrix, the source vector, their CentDer derivatives and the TauStep steps;
// CentDer of the full matrix is taken through its 6 distinct elements (CentDer commutes with negation
// exactly and maps the zero diagonal to zero).  k_stokes_thr (plane-parallel) and k_stokes_sph (spherical
// rays of up to 2 ntau points) give every thread one (wavelength, angle) sweep over per-thread work
// arrays in global memory.
// ================================================================================================
#define STK_FIELDS 22   // per depth: PhiI, 6 K, 6 KD, 4 SRC4, 4 SRD, Deltau

__device__ __forceinline__ void centder_pt(const double *D, const double *Y, int stride, int N, int k, double *out) {
    // Yp at 0-based depth k for one component with values Y[t * stride]
    if (k == 0) { *out = (Y[stride] - Y[0]) / D[0]; return; }
    if (k == N - 1) { *out = (Y[(N - 1) * stride] - Y[(N - 2) * stride]) / D[N - 2]; return; }
    double Dx = D[k - 1], Dx1 = D[k];
    double InvDx = 1.0 / Dx, InvDx1 = 1.0 / Dx1;
    double Lambda = (1.0 + Dx1 / (Dx + Dx1)) / 3.0, Lambda1 = 1.0 - Lambda;
    double Der = (Y[k * stride] - Y[(k - 1) * stride]) * InvDx, Der1 = (Y[(k + 1) * stride] - Y[k * stride]) * InvDx1;
    *out = (Der * Der1 > 0.0) ? (Der / (Lambda * Der1 + Lambda1 * Der)) * Der1 : 0.0;
}

// Gaussian elimination with row pivoting (Solve4x4, solver.f90:541-588)
__device__ __forceinline__ void solve4x4(double (&M)[4][4], double (&R)[4], double (&X)[4]) {
    double ip[4];
#pragma unroll
    for (int k = 0; k < 4; k++) {
        if (k < 3) {
            int piv = k;
            double p = fabs(M[k][k]);
#pragma unroll
            for (int i = k + 1; i < 4; i++) if (fabs(M[i][k]) > p) { p = fabs(M[i][k]); piv = i; }
#pragma unroll
            for (int i = k + 1; i < 4; i++)
                if (piv == i) {
#pragma unroll
                    for (int j = k; j < 4; j++) { const double sw = M[k][j]; M[k][j] = M[i][j]; M[i][j] = sw; }
                    const double sw = R[k]; R[k] = R[i]; R[i] = sw;
                }
        }
        ip[k] = rcp64(M[k][k]);
#pragma unroll
        for (int i = k + 1; i < 4; i++) {
            const double f = M[i][k] * ip[k];
#pragma unroll
            for (int j = k + 1; j < 4; j++) M[i][j] = fma(-f, M[k][j], M[i][j]);
            R[i] = fma(-f, R[k], R[i]);
        }
    }
#pragma unroll
    for (int k = 3; k >= 0; k--) {
        double r = R[k];
#pragma unroll
        for (int j = k + 1; j < 4; j++) r = fma(-M[k][j], X[j], r);
        X[k] = r * ip[k];
    }
}

// The propagation matrix of one point (solver.f90:311-326) by its 6 distinct elements: symmetric in the first
// row and column (Q, U, V absorption), antisymmetric below (dispersion), zero diagonal.
struct PropK {
    double a, b, c, q, u, v;             // PhiQ, PhiU, PhiV, PsiQ, PsiU, PsiV
    // K x
    __device__ __forceinline__ void mul(const double (&x)[4], double (&y)[4]) const {
        y[0] = fma(a, x[1], fma(b, x[2], c * x[3]));
        y[1] = fma(a, x[0], fma(v, x[2], -(u * x[3])));
        y[2] = fma(b, x[0], fma(-v, x[1], q * x[3]));
        y[3] = fma(c, x[0], fma(u, x[1], -(q * x[2])));
    }
    // element (i, j)
    __device__ __forceinline__ double at(int i, int j) const {
        const double t[4][4] = { { 0.0, a, b, c }, { a, 0.0, v, -u }, { b, -v, 0.0, q }, { c, u, -q, 0.0 } };
        return t[i][j];
    }
};

// K K + K' of a point: ten distinct values of K K, K' of K's own form
__device__ __forceinline__ void prop_square(const PropK &k, const PropK &d, double (&X)[4][4]) {
    const double aa = k.a * k.a, bb = k.b * k.b, cc = k.c * k.c, qq = k.q * k.q, uu = k.u * k.u, vv = k.v * k.v;
    const double s12 = fma(k.a, k.b, k.u * k.q), s13 = fma(k.a, k.c, k.v * k.q), s23 = fma(k.b, k.c, k.v * k.u);
    const double n01 = fma(k.c, k.u, -(k.b * k.v)), n02 = fma(k.a, k.v, -(k.c * k.q)), n03 = fma(k.b, k.q, -(k.a * k.u));
    X[0][0] = aa + bb + cc; X[1][1] = aa - vv - uu; X[2][2] = bb - vv - qq; X[3][3] = cc - uu - qq;
    X[0][1] = d.a + n01; X[1][0] = d.a - n01;
    X[0][2] = d.b + n02; X[2][0] = d.b - n02;
    X[0][3] = d.c + n03; X[3][0] = d.c - n03;
    X[1][2] = s12 + d.v; X[2][1] = s12 - d.v;
    X[1][3] = s13 - d.u; X[3][1] = s13 + d.u;
    X[2][3] = s23 + d.q; X[3][2] = s23 - d.q;
}

// The DELO-Bezier sweep of StokesPrfPP / StokesPrfSph (solver.f90:341-390, 486-534) over the N points of
// one ray, run by one thread from per-point fields (field-major, leading dimension ld, element stride es):
// Kv / KD the 6 distinct propagation elements and their derivatives, SRC4 / SRD the source vector and its
// derivative, Dt the optical-depth steps.  XINT2 holds the boundary Stokes vector on entry and the emergent one
// on return.  With G = Gamma Dtau/2 and Q = K K + K' the step (solver.f90:360-388) is
//   [1 + (Alpha + Gamma (Dtau/2 + 1)) K0 + G Q0] I0 = Eps I1 + G Q1 I1 + K1 [(Gamma (Dtau/2 - 1) - Beta) I1 - G S1]
//                    + (Beta + Gamma) S1 + (Alpha + Gamma) S0 + G (K0 S0 + S0' - S1')
// in which K's form leaves 12 products of each K x and 18 of K K.
__device__ __forceinline__ void stokes_sweep(int N, int ld, const double *Kv, const double *KD, const double *SRC4,
                                             const double *SRD, const double *Dt, double (&XINT2)[4], size_t es = 1) {
    auto prop = [&](const double *f, int k) {
        return PropK{ f[k * es], f[(ld + k) * es], f[((size_t)2 * ld + k) * es], f[((size_t)3 * ld + k) * es],
                      f[((size_t)4 * ld + k) * es], f[((size_t)5 * ld + k) * es] };
    };
    PropK K1 = prop(Kv, N - 1);
    double Q1[4][4], S1[4], D1[4];
    prop_square(K1, prop(KD, N - 1), Q1);
#pragma unroll
    for (int i = 0; i < 4; i++) { S1[i] = SRC4[((size_t)i * ld + N - 1) * es]; D1[i] = SRD[((size_t)i * ld + N - 1) * es]; }
    for (int k = N - 2; k >= 0; k--) {
        const PropK K0 = prop(Kv, k), KD0 = prop(KD, k);
        const double Dtau = Dt[k * es], h = 0.5 * Dtau;
        double Eps, Alpha, Beta, Gamma, S0[4], D0[4];
#pragma unroll
        for (int i = 0; i < 4; i++) { S0[i] = SRC4[((size_t)i * ld + k) * es]; D0[i] = SRD[((size_t)i * ld + k) * es]; }
        delo_coef(Dtau, Eps, Alpha, Beta, Gamma);
        Gamma = Gamma * 0.5;
        const double G = Gamma * h, c1 = fma(Gamma, h - 1.0, -Beta), c0 = fma(Gamma, h + 1.0, Alpha);
        double w[4], y[4], z[4], R[4];
#pragma unroll
        for (int i = 0; i < 4; i++) w[i] = fma(c1, XINT2[i], -(G * S1[i]));
        K1.mul(w, y);
        K0.mul(S0, z);
#pragma unroll
        for (int i = 0; i < 4; i++) {
            double m = 0.0;
#pragma unroll
            for (int j = 0; j < 4; j++) m = fma(Q1[i][j], XINT2[j], m);
            R[i] = fma(Eps, XINT2[i], y[i]) + fma(Beta + Gamma, S1[i], (Alpha + Gamma) * S0[i]) +
                   G * (m + z[i] + (D0[i] - D1[i]));
        }
        double M[4][4];
        prop_square(K0, KD0, Q1);
#pragma unroll
        for (int i = 0; i < 4; i++)
#pragma unroll
            for (int j = 0; j < 4; j++)
                M[i][j] = i == j ? fma(G, Q1[i][j], 1.0) : fma(c0, K0.at(i, j), G * Q1[i][j]);
        solve4x4(M, R, XINT2);
        K1 = K0;
#pragma unroll
        for (int i = 0; i < 4; i++) { S1[i] = S0[i]; D1[i] = D0[i]; }
    }
}

// propagation matrix elements normalised by PhiI and the source vector at one point (solver.f90:296-330,
// 431-465): m = MagLineOpac(:, ia), g = (SPhi2, CPhi2, CPhi, S2Psi, C2Psi); returns PhiI
__device__ __forceinline__ double stokes_point(const double *m, double lop, double cop, double sr, const double *g,
                                               double *e6, double *s4) {
    double Php = m[0], Phb = m[1], Phr = m[2], Psp = m[3], Psb = m[4], Psr = m[5];
    double SPhi2 = g[0], CPhi2 = g[1], CPhi = g[2], S2Psi = g[3], C2Psi = g[4];
    double PI = 0.5 * (Php * SPhi2 + 0.5 * (Phr + Phb) * (1.0 + CPhi2)) + lop + cop;
    double InvPhiI = 1.0 / PI;
    double Sabs = 0.5 * (Php - 0.5 * (Phr + Phb)) * SPhi2;
    double PhiQ = Sabs * C2Psi * InvPhiI, PhiU = Sabs * S2Psi * InvPhiI;
    double PhiV = 0.5 * (Phr - Phb) * CPhi * InvPhiI;
    double Sdis = 0.5 * (Psp - 0.5 * (Psr + Psb)) * SPhi2;
    double PsiQ = Sdis * C2Psi * InvPhiI, PsiU = Sdis * S2Psi * InvPhiI;
    double PsiV = 0.5 * (Psr - Psb) * CPhi * InvPhiI;
    e6[0] = PhiQ; e6[1] = PhiU; e6[2] = PhiV; e6[3] = PsiQ; e6[4] = PsiU; e6[5] = PsiV;
    s4[0] = sr; s4[1] = sr * PhiQ; s4[2] = sr * PhiU; s4[3] = sr * PhiV;
    return PI;
}

// StokesPrfPP, one thread per (wavelength, angle) from the first wavelength iwl0 on, in two launches
// over per-thread global work arrays (STK_FIELDS x ntau doubles, element stride = the launch's thread
// count T, so that the threads of a warp touch consecutive addresses).  k_stokes_prep builds the
// propagation data, TauStep and CentDer over depth: a thread takes a run of depths (blockIdx.y) with the
// points, steps and slopes around the present one in registers, so each field is written once and nothing is
// read back; k_stokes_thr runs the sequential 4x4 sweep, every lane of every warp.  Bound by the traffic of
// the 21 fields (8.5 GB of 50,001 wavelengths x 9 angles x 56 depths, there and back): 2.1 ms, against 6.2 ms
// when the steps and slopes were formed from fields written before.
#define STK_RUNS 4
__global__ void __launch_bounds__(128)
k_stokes_prep(AtmView A, const double *__restrict__ lineopac, const double *__restrict__ mlo,
              const double *__restrict__ rhox, int nmu, const double *__restrict__ xmu,
              const double *__restrict__ geo, int iwl0, int nwl_chunk, double *work) {
    const size_t T = (size_t)gridDim.x * blockDim.x;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nwl_chunk * nmu) return;
    const int iwl = iwl0 + g / nmu, im = g - (g / nmu) * nmu;
    const int N = A.ntau, run = (N + STK_RUNS - 1) / STK_RUNS, ta = blockIdx.y * run, tb = min(ta + run, N);
    if (ta >= tb) return;
    double *W = work + g;
#define F(f, t) W[((size_t)(f) * N + (t)) * T]
    const double PlkC1 = FSG_HC * FSG_VC * 1e13 / FSG_KBOLT;
    const double wl = A.wave[iwl] + A.wfirst;
    const double C1 = PlkC1 / wl, C2 = exp(50.7649141 - 5.0 * log(wl));
    const double gm[5] = { geo[0 * nmu + im], geo[1 * nmu + im], geo[2 * nmu + im], geo[3 * nmu + im],
                           geo[4 * nmu + im] };
    const double imu = 1.0 / xmu[im];
    // the point at depth t: PhiI, then y = the 6 elements and the source vector
    auto point = [&](int t, double (&y)[10]) {
        const size_t o = (size_t)iwl * N + t;
        const double sr = C2 / (exp(C1 / A.xi[XI_T * N + t]) - 1.0);
        double e6[6], s4[4];
        const double p = stokes_point(mlo + o * 6, lineopac[o], A.contopac[o], sr, gm, e6, s4);
#pragma unroll
        for (int q = 0; q < 6; q++) y[q] = e6[q];
#pragma unroll
        for (int q = 0; q < 4; q++) y[6 + q] = s4[q];
        return p;
    };
    // TauStep (solver.f90:591-615) from depth t to t + 1 with Xmu(im), given the slopes of PhiI behind and before
    auto step = [&](int t) { return (rhox[t + 1] - rhox[t]) * imu; };
    auto tau = [&](int t, double p0, double p1, double sa, double sb) {
        const double dx = step(t), yp = t == 0 ? sb : hmean(sa, sb, lambda_of(step(t - 1), dx));
        return dx * (p1 + 2.0 * p0 + dx * 0.5 * yp) * (1.0 / 3.0);
    };
    double y0[10], y1[10], gp[10];        // point t, point t + 1, slopes over the step before t
    double p0, p1, sa = 0.0, dprev = 0.0;
    if (ta > 0) {
        double ym[10], yq[10];
        const double pm = point(ta - 1, ym);
        p0 = point(ta, y0);
        sa = (p0 - pm) * rcp64(step(ta - 1));
        const double sq = ta > 1 ? (pm - point(ta - 2, yq)) * rcp64(step(ta - 2)) : 0.0;
        dprev = tau(ta - 1, pm, p0, sq, sa);
        const double id = rcp64_step(dprev);
#pragma unroll
        for (int q = 0; q < 10; q++) gp[q] = (y0[q] - ym[q]) * id;
    } else {
        p0 = point(0, y0);
    }
    for (int t = ta; t < tb; t++) {
        // CentDer (solver.f90:618-647) of every component at t from the slopes on either side
        double out[10], d = 0.0;
        if (t < N - 1) {
            p1 = point(t + 1, y1);
            const double sb = (p1 - p0) * rcp64(step(t));
            d = tau(t, p0, p1, sa, sb);
            F(21, t) = d;
            const double id = rcp64_step(d), lam = t > 0 ? lambda_of(dprev, d) : 0.0;
#pragma unroll
            for (int q = 0; q < 10; q++) {
                const double gn = (y1[q] - y0[q]) * id;
                out[q] = t > 0 ? hmean(gp[q], gn, lam) : gn;
                gp[q] = gn;
            }
            sa = sb;
        } else {
#pragma unroll
            for (int q = 0; q < 10; q++) out[q] = gp[q];
        }
#pragma unroll
        for (int q = 0; q < 6; q++) { F(1 + q, t) = y0[q]; F(7 + q, t) = out[q]; }
#pragma unroll
        for (int q = 0; q < 4; q++) { F(13 + q, t) = y0[6 + q]; F(17 + q, t) = out[6 + q]; }
        p0 = p1; dprev = d;
#pragma unroll
        for (int q = 0; q < 10; q++) y0[q] = y1[q];
    }
#undef F
}

__global__ void __launch_bounds__(128)
k_stokes_thr(AtmView A, int nmu, int iwl0, int nwl_chunk, const double *work, double *spz) {
    const size_t T = (size_t)gridDim.x * blockDim.x;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nwl_chunk * nmu) return;
    const int iwl = iwl0 + g / nmu, im = g - (g / nmu) * nmu;
    const int N = A.ntau;
    const double *W = work + g;
#define F(f, t) W[((size_t)(f) * N + (t)) * T]
    double XINT2[4] = { F(13, N - 1), 0.0, 0.0, 0.0 };
    stokes_sweep(N, N, &F(1, 0), &F(7, 0), &F(13, 0), &F(17, 0), &F(21, 0), XINT2, T);
    for (int q = 0; q < 4; q++) spz[((size_t)iwl * 4 + q) * nmu + im] = XINT2[q];
#undef F
}

// StokesPrfSph (solver.f90:402-538), one thread per (wavelength, ray) from the first wavelength iwl0
// on, with per-thread work arrays as k_stokes_thr (up to 2 ntau points per ray).  Each point gathers the
// six profiles, line and continuum opacity and source of the layer it samples, with the field
// projection of that point (geo [5][nmu][stride]); TauStep runs on the ray's column mass (mu = 1); the
// sweep starts from zero incoming light for grazing rays, Src(N) otherwise.
__global__ void __launch_bounds__(128)
k_stokes_sph(AtmView A, const double *__restrict__ lineopac, const double *__restrict__ mlo, RayView R,
             const double *__restrict__ geo, int iwl0, int nwl_chunk, double *work, double *spz) {
    const size_t T = (size_t)gridDim.x * blockDim.x;
    const int nmu = R.nmu, M = R.stride, nt = A.ntau;
    const int g = blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= nwl_chunk * nmu) return;
    const int iwl = iwl0 + g / nmu, im = g - (g / nmu) * nmu;
    const int N = R.n[im];
    const int *mp = R.map + (size_t)im * M;
    const double *m = R.m + (size_t)im * M;
    double *W = work + g;
#define F(f, t) W[((size_t)(f) * M + (t)) * T]
    const double PlkC1 = FSG_HC * FSG_VC * 1e13 / FSG_KBOLT;
    const double wl = A.wave[iwl] + A.wfirst;
    const double C1 = PlkC1 / wl, C2 = exp(50.7649141 - 5.0 * log(wl));
    const size_t gs = (size_t)nmu * M, go = (size_t)im * M;
    for (int t = 0; t < N; t++) {
        const int ia = mp[t];
        const size_t o = (size_t)iwl * nt + ia;
        const double sr = C2 / (exp(C1 / A.xi[XI_T * nt + ia]) - 1.0);
        const double gm[5] = { geo[go + t], geo[gs + go + t], geo[2 * gs + go + t], geo[3 * gs + go + t],
                               geo[4 * gs + go + t] };
        double e6[6], s4[4];
        F(0, t) = stokes_point(mlo + o * 6, lineopac[o], A.contopac[o], sr, gm, e6, s4);
        for (int q = 0; q < 6; q++) F(1 + q, t) = e6[q];
        for (int q = 0; q < 4; q++) F(13 + q, t) = s4[q];
    }
    // TauStep (solver.f90:591-615) on the ray's column mass
    for (int t = 0; t < N - 1; t++) {
        if (t == 0) {
            double Dx1 = m[1] - m[0], Yp = (F(0, 1) - F(0, 0)) / Dx1;
            F(21, 0) = Dx1 * (F(0, 1) + 2.0 * F(0, 0) + Dx1 / 2.0 * Yp) / 3.0;
        } else {
            double Dx = m[t] - m[t - 1], Dx1 = m[t + 1] - m[t];
            double Der = (F(0, t) - F(0, t - 1)) / Dx, Der1 = (F(0, t + 1) - F(0, t)) / Dx1, Yp;
            if (Der * Der1 > 0.0) {
                double Lambda = (1.0 + Dx1 / (Dx + Dx1)) / 3.0;
                Yp = (Der / (Lambda * Der1 + (1.0 - Lambda) * Der)) * Der1;
            } else Yp = 0.0;
            F(21, t) = Dx1 * (F(0, t + 1) + 2.0 * F(0, t) + Dx1 / 2.0 * Yp) / 3.0;
        }
    }
    // CentDer (solver.f90:618-647) of SRC4 (fields 13-16 -> 17-20) and of the 6 elements (1-6 -> 7-12)
    for (int row = 0; row < 10; row++) {
        const int fi = row < 4 ? 13 + row : 1 + (row - 4), fo = row < 4 ? 17 + row : 7 + (row - 4);
        for (int k = 0; k < N; k++) {
            double out;
            if (k == 0) out = (F(fi, 1) - F(fi, 0)) / F(21, 0);
            else if (k == N - 1) out = (F(fi, N - 1) - F(fi, N - 2)) / F(21, N - 2);
            else {
                double Dx = F(21, k - 1), Dx1 = F(21, k);
                double InvDx = 1.0 / Dx, InvDx1 = 1.0 / Dx1;
                double Lambda = (1.0 + Dx1 / (Dx + Dx1)) / 3.0, Lambda1 = 1.0 - Lambda;
                double Der = (F(fi, k) - F(fi, k - 1)) * InvDx, Der1 = (F(fi, k + 1) - F(fi, k)) * InvDx1;
                out = (Der * Der1 > 0.0) ? (Der / (Lambda * Der1 + Lambda1 * Der)) * Der1 : 0.0;
            }
            F(fo, k) = out;
        }
    }
    double XINT2[4] = { R.graz[im] ? 0.0 : F(13, N - 1), 0.0, 0.0, 0.0 };
    stokes_sweep(N, M, &F(1, 0), &F(7, 0), &F(13, 0), &F(17, 0), &F(21, 0), XINT2, T);
    for (int q = 0; q < 4; q++) spz[((size_t)iwl * 4 + q) * nmu + im] = XINT2[q];
#undef F
}

// Stokes-I flux of the spherical path: Sf = sum over mu of SpZ(mu, 1) Wmu (convol.f90:233-234)
__global__ void k_stokes_flux(int nwl, int nmu, const double *__restrict__ spz, const double *__restrict__ wmu,
                              double *sfl) {
    int iwl = blockIdx.x * blockDim.x + threadIdx.x;
    if (iwl >= nwl) return;
    double a = 0.0;
    for (int q = 0; q < nmu; q++) a = a + spz[(size_t)iwl * 4 * nmu + q] * wmu[q];
    sfl[iwl] = a;
}

// ================================================================================================
// host drivers
// ================================================================================================
struct fsg_ctx;
AtmView fsg_view(const fsg_ctx *ctx);

// per-thread work arrays of k_stokes_thr for one chunk of nwl_chunk wavelengths
size_t fsg_stokes_work(int nt, int nmu, int nwl_chunk) {
    const size_t nthr = ((size_t)nwl_chunk * nmu + 127) / 128 * 128;
    return sizeof(double) * STK_FIELDS * (size_t)nt * nthr;
}

// the most wavelengths (at least 1, at most nwl) whose work arrays fit in max_bytes
int fsg_stokes_chunk(int nt, int nmu, int nwl, size_t max_bytes) {
    const size_t per_wl = sizeof(double) * STK_FIELDS * (size_t)nt * nmu;
    size_t c = max_bytes / per_wl;
    if (c > (size_t)nwl) c = (size_t)nwl;
    return c < 1 ? 1 : (int)c;
}

// StokesPrfPP over the grid: k_stokes_thr in chunks of nwl_chunk wavelengths whose work arrays fit `work`
// (fsg_stokes_work bytes), then the Stokes-I flux.
int fsg_launch_stokes(cudaStream_t s, const AtmView &A, const double *lineopac, const double *mlo, const double *rhox,
                      int nmu, const double *xmu, const double *wmu, const double *geo, double *spz, double *sfl,
                      double *work, int nwl_chunk) {
    if (nwl_chunk < 1) return FSG_E_ARG;
    for (int w0 = 0; w0 < A.nwl; w0 += nwl_chunk) {
        const int nw = std::min(nwl_chunk, A.nwl - w0);
        const int nb = (nwl_chunk * nmu + 127) / 128;      // the grid of a full chunk: fixed element stride
        k_stokes_prep<<<dim3(nb, STK_RUNS), 128, 0, s>>>(A, lineopac, mlo, rhox, nmu, xmu, geo, w0, nw, work);
        k_stokes_thr<<<nb, 128, 0, s>>>(A, nmu, w0, nw, work, spz);
    }
    if (sfl) k_stokes_flux<<<(A.nwl + 127) / 128, 128, 0, s>>>(A.nwl, nmu, spz, wmu, sfl);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

int fsg_launch_stokes_sph(cudaStream_t s, const AtmView &A, const double *lineopac, const double *mlo,
                          const RayView &R, const double *wmu, const double *geo, double *spz, double *sfl,
                          double *work, int nwl_chunk) {
    if (nwl_chunk < 1) return FSG_E_ARG;
    for (int w0 = 0; w0 < A.nwl; w0 += nwl_chunk) {
        const int nw = std::min(nwl_chunk, A.nwl - w0);
        const int nb = (nwl_chunk * R.nmu + 127) / 128;     // the grid of a full chunk: fixed element stride
        k_stokes_sph<<<nb, 128, 0, s>>>(A, lineopac, mlo, R, geo, w0, nw, work, spz);
    }
    if (sfl) k_stokes_flux<<<(A.nwl + 127) / 128, 128, 0, s>>>(A.nwl, R.nmu, spz, wmu, sfl);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

void fsg_launch_mag_center(cudaStream_t s, const AtmView &A, const LineView &L, const ZView &Z, double Bsplit,
                           const VoigtTables &T, int32_t *flags, int32_t *ileft, int32_t *iright,
                           unsigned long long *nkeep) {
    if (L.n > 0)
        k_mag_center<<<(unsigned)((L.n + 3) / 4), 128, 0, s>>>(A, L, Z, Bsplit, T.vtab, T.anode, T.aida, flags, ileft,
                                                                iright, nkeep);
}

// ================================================================================================
// MagLineOpacity1 and StokesPrfPP on their own, batched (kernel-level entry points)
// ================================================================================================
// MagLineOpacity1 (opacity.f90:391-464) at npts points; the block's Zeeman components are indexed by
// line (Z's CSR arrays); one warp per point, lanes over depths; out [npts][ntau][6]
__global__ void k_mag_lineopacity1_pts(AtmView A, BlockView B, ZView Z, int64_t npts, const double *__restrict__ wl,
                                       const int32_t *__restrict__ l1, const int32_t *__restrict__ l2,
                                       const int32_t *__restrict__ iwl, int64_t loff, const float2 *__restrict__ fvtab,
                                       const double *__restrict__ anode, const double *__restrict__ aida, double *out) {
    const int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (k >= npts) return;
    const int nt = A.ntau;
    for (int t = lane; t < nt; t += 32) {
        double m[6] = { 0, 0, 0, 0, 0, 0 };
        for (int64_t il = l1[k]; il <= l2[k]; il++) {
            const int f = B.flags[il - 1];
            if ((f & FSG_F_WEAK) || (f & FSG_F_WIDE) || iwl[k] < B.ileft[il - 1] || iwl[k] > B.iright[il - 1]) continue;
            const size_t o = (size_t)(il - loff - 1) * nt + t;
            mag_profiles_t(A, t, wl[k], B.wlcent[il - 1], (f >> 8) & 255, Z, il - 1, B.cop[o], B.vv[o], B.av[o],
                           fvtab, anode, aida, m);
        }
        double *dst = out + ((size_t)k * nt + t) * 6;
        for (int q = 0; q < 6; q++) dst[q] = (A.motype == 1) ? m[q] / A.contstd[t] : m[q];
    }
}

// StokesPrfPP (solver.f90:265-394) at the grid wavelengths iwl[k] (1-based) with given source functions
// src [npts][ntau]: one thread per (point, angle) over per-thread work arrays, as k_stokes_thr;
// geo [5][nmu] (SPhi2, CPhi2, CPhi, S2Psi, C2Psi); out [npts][4][nmu]
__global__ void __launch_bounds__(128)
k_stokes_prf_pts(AtmView A, const double *__restrict__ lineopac, const double *__restrict__ mlo,
                 const double *__restrict__ rhox, int nmu, const double *__restrict__ xmu,
                 const double *__restrict__ geo, int64_t npts, const int32_t *__restrict__ iwls,
                 const double *__restrict__ src, double *work, double *out) {
    const size_t T = (size_t)gridDim.x * blockDim.x;
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= npts * nmu) return;
    const int64_t k = g / nmu;
    const int im = (int)(g - k * nmu);
    const int iwl = iwls[k] - 1;
    const int N = A.ntau;
    double *W = work + g;
#define F(f, t) W[((size_t)(f) * N + (t)) * T]
    const double gm[5] = { geo[0 * nmu + im], geo[1 * nmu + im], geo[2 * nmu + im], geo[3 * nmu + im],
                           geo[4 * nmu + im] };
    for (int t = 0; t < N; t++) {
        const size_t o = (size_t)iwl * N + t;
        double e6[6], s4[4];
        F(0, t) = stokes_point(mlo + o * 6, lineopac[o], A.contopac[o], src[(size_t)k * N + t], gm, e6, s4);
        for (int q = 0; q < 6; q++) F(1 + q, t) = e6[q];
        for (int q = 0; q < 4; q++) F(13 + q, t) = s4[q];
    }
    const double Xmu = xmu[im];
    for (int t = 0; t < N - 1; t++) {
        if (t == 0) {
            double Dx1 = (rhox[1] - rhox[0]) / Xmu;
            double Yp = (F(0, 1) - F(0, 0)) / Dx1;
            F(21, 0) = Dx1 * (F(0, 1) + 2.0 * F(0, 0) + Dx1 / 2.0 * Yp) / 3.0;
        } else {
            const int kk = t + 1;
            double Dx = (rhox[kk - 1] - rhox[kk - 2]) / Xmu, Dx1 = (rhox[kk] - rhox[kk - 1]) / Xmu;
            double Der = (F(0, kk - 1) - F(0, kk - 2)) / Dx, Der1 = (F(0, kk) - F(0, kk - 1)) / Dx1, Yp;
            if (Der * Der1 > 0.0) {
                double Lambda = (1.0 + Dx1 / (Dx + Dx1)) / 3.0;
                Yp = (Der / (Lambda * Der1 + (1.0 - Lambda) * Der)) * Der1;
            } else Yp = 0.0;
            F(21, kk - 1) = Dx1 * (F(0, kk) + 2.0 * F(0, kk - 1) + Dx1 / 2.0 * Yp) / 3.0;
        }
    }
    for (int row = 0; row < 10; row++) {
        const int fi = row < 4 ? 13 + row : 1 + (row - 4), fo = row < 4 ? 17 + row : 7 + (row - 4);
        for (int kk = 0; kk < N; kk++) {
            double o;
            if (kk == 0) o = (F(fi, 1) - F(fi, 0)) / F(21, 0);
            else if (kk == N - 1) o = (F(fi, N - 1) - F(fi, N - 2)) / F(21, N - 2);
            else {
                double Dx = F(21, kk - 1), Dx1 = F(21, kk);
                double InvDx = 1.0 / Dx, InvDx1 = 1.0 / Dx1;
                double Lambda = (1.0 + Dx1 / (Dx + Dx1)) / 3.0, Lambda1 = 1.0 - Lambda;
                double Der = (F(fi, kk) - F(fi, kk - 1)) * InvDx, Der1 = (F(fi, kk + 1) - F(fi, kk)) * InvDx1;
                o = (Der * Der1 > 0.0) ? (Der / (Lambda * Der1 + Lambda1 * Der)) * Der1 : 0.0;
            }
            F(fo, kk) = o;
        }
    }
    double XINT2[4] = { F(13, N - 1), 0.0, 0.0, 0.0 };
    stokes_sweep(N, N, &F(1, 0), &F(7, 0), &F(13, 0), &F(17, 0), &F(21, 0), XINT2, T);
    for (int q = 0; q < 4; q++) out[((size_t)k * 4 + q) * nmu + im] = XINT2[q];
#undef F
}

void fsg_launch_mag_lineopacity1_pts(cudaStream_t s, const AtmView &A, const BlockView &B, const ZView &Z,
                                     int64_t npts, const double *wl, const int32_t *l1, const int32_t *l2,
                                     const int32_t *iwl, int64_t loff, const VoigtTables &T, double *out) {
    if (npts > 0)
        k_mag_lineopacity1_pts<<<(unsigned)((npts + 7) / 8), 256, 0, s>>>(A, B, Z, npts, wl, l1, l2, iwl, loff,
                                                                          T.fvtab, T.anode, T.aida, out);
}

size_t fsg_stokes_pts_work(int64_t npts, int nmu, int ntau) {
    const int64_t thr = ((npts * nmu + 127) / 128) * 128;
    return sizeof(double) * (size_t)STK_FIELDS * (size_t)ntau * (size_t)thr;
}

void fsg_launch_stokes_prf_pts(cudaStream_t s, const AtmView &A, const double *lineopac, const double *mlo,
                               const double *rhox, int nmu, const double *xmu, const double *geo, int64_t npts,
                               const int32_t *iwl, const double *src, double *work, double *out) {
    const int64_t m = npts * nmu;
    if (m > 0)
        k_stokes_prf_pts<<<(unsigned)((m + 127) / 128), 128, 0, s>>>(A, lineopac, mlo, rhox, nmu, xmu, geo, npts, iwl,
                                                                     src, work, out);
}
