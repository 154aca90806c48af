// fsg_solve.cu -- the scalar formal solver (built -fmad=false; fused operations are written out).
//
//   k_radtran       RadTranCalc (synth.f90:1825-1866) + DiskInteg quadrature (convol.f90:233-234)
//   k_radtran_sph   RadTranCalc for spherical models (synth.f90:1868-1898): LocPrfSph along each ray
//   k_linstr        LinStrCalc (synth.f90:1774-1822), both geometries
//
// A CTA takes SOLVE_C columns (wavelengths; for k_linstr line centres): their continuum and continuum + line
// opacities and Planck source go to shared memory, then one thread per (column, kind, angle) sweeps the
// depths.  Plane-parallel models share TauStep, CentDer and the Bezier term over the angles, worked out with
// threads over depths first; the steps of a spherical ray are its own and are formed as the sweep reaches them.
//
// Bound by the FP64 pipe: a sweep step is an exponential, a reciprocal and some 25 operations, and there are
// 2 nmu of them per column and depth.  So divisions are reciprocals (rcp64) times the numerator, constants are
// multiplied, quantities of the depth scale alone are formed once per CTA, and the two DELO branches are
// entered only by warps that need them.  482,832 wavelengths x 71 depths x 7 angles: 2.6 ms (5.6 ms when every
// step divided and the Taylor branch's eight divisions were paid beside the exponential); 40,001 wavelengths x 7 rays
// through a spherical model 0.30 ms (0.63); the central depths of 20,000 lines 0.13 ms (0.89 with a thread per line).
#include "fsg_fp64.cuh"

#define SOLVE_C 8

// one step of the sweep (solver.f90:139-142): Y Eps + Alpha y0 + Beta y1 + Gamma u
__device__ __forceinline__ double delo_step(double d, double Y, double y0, double y1, double u) {
    double Eps, Al, Be, Ga;
    delo_coef(d, Eps, Al, Be, Ga);
    return fma(Y, Eps, fma(Al, y0, fma(Be, y1, Ga * u)));
}

// CentDer (solver.f90:618-647) of y on the scale of the steps d, at point t of nt
__device__ __forceinline__ double centder_at(const double *d, const double *y, int nt, int t) {
    if (t == 0) return (y[1] - y[0]) * rcp64_step(d[0]);
    if (t == nt - 1) return (y[nt - 1] - y[nt - 2]) * rcp64_step(d[nt - 2]);
    const double dx = d[t - 1], dx1 = d[t];
    return hmean((y[t] - y[t - 1]) * rcp64_step(dx), (y[t + 1] - y[t]) * rcp64_step(dx1), lambda_of(dx, dx1));
}

// shared memory of a CTA: source S[c][ld], opacities X[kind][c][ld] (later the Bezier terms), steps
// D[kind][c][ld], intensities I[kind][c][nmu], 1 / step and Lambda of the depth scale [nt].  ld is odd, so
// that the columns a warp sweeps lie in different banks.
struct Columns {
    double *S, *X, *D, *I, *idx, *lam;
    int ld;
};
__host__ __device__ inline int column_ld(int nt) { return nt | 1; }
static size_t columns_smem(int nt, int nmu) {
    return sizeof(double) * ((size_t)5 * SOLVE_C * column_ld(nt) + 2 * SOLVE_C * nmu + 2 * nt);
}
__device__ __forceinline__ Columns columns(double *sm, int nt, int nmu) {
    Columns C;
    C.ld = column_ld(nt);
    C.S = sm; C.X = C.S + SOLVE_C * C.ld; C.D = C.X + 2 * SOLVE_C * C.ld; C.I = C.D + 2 * SOLVE_C * C.ld;
    C.idx = C.I + 2 * SOLVE_C * nmu; C.lam = C.idx + nt;
    return C;
}
static int columns_threads(int nmu) {                  // a thread per sweep, 128 at least
    const int n = 2 * SOLVE_C * nmu;
    return n <= 128 ? 128 : (n + 31) / 32 * 32;
}

// Planck source at wl (the source function of RadTranCalc) from C1 = hc / (k wl) and C2
__device__ __forceinline__ double planck(double C1, double C2, double T) { return C2 / (exp(C1 / T) - 1.0); }

// LocPrfPP (solver.f90:123-179) of the first nw columns, kinds k0 .. 1 (0 continuum, 1 with lines): the
// emergent intensities to C.I.  Every thread of the CTA, after the barrier that completes C.S and C.X.
__device__ __forceinline__ void solve_pp(const Columns &C, int nt, int nw, int nk, int nmu,
                                         const double *__restrict__ rhox, const double *__restrict__ xmu) {
    const int ld = C.ld;
    for (int t = threadIdx.x; t < nt - 1; t += blockDim.x) {
        const double dx1 = rhox[t + 1] - rhox[t];
        C.idx[t] = 1.0 / dx1;
        C.lam[t] = t > 0 ? (1.0 + dx1 / (rhox[t] - rhox[t - 1] + dx1)) / 3.0 : 0.0;
    }
    __syncthreads();
    // TauStep at mu = 1 (solver.f90:591-615)
    for (int e = threadIdx.x; e < nk * nw * nt; e += blockDim.x) {
        const int kw = e / nt, t = e - kw * nt, col = (kw / nw) * SOLVE_C + kw % nw;
        const double *x = C.X + col * ld;
        double d = 0.0;
        if (t < nt - 1) {
            const double dx1 = rhox[t + 1] - rhox[t], der1 = (x[t + 1] - x[t]) * C.idx[t];
            const double yp = t == 0 ? der1 : hmean((x[t] - x[t - 1]) * C.idx[t - 1], der1, C.lam[t]);
            d = dx1 * (x[t + 1] + 2.0 * x[t] + dx1 * 0.5 * yp) * (1.0 / 3.0);
        }
        C.D[col * ld + t] = d;
    }
    __syncthreads();
    // Bezier control term (solver.f90:136-138) from CentDer of the source, over the opacities
    for (int e = threadIdx.x; e < nk * nw * nt; e += blockDim.x) {
        const int kw = e / nt, t = e - kw * nt, w = kw % nw, col = (kw / nw) * SOLVE_C + w;
        if (t >= nt - 1) continue;
        const double *d = C.D + col * ld, *y = C.S + w * ld;
        const double r0 = centder_at(d, y, nt, t), r1 = centder_at(d, y, nt, t + 1);
        C.X[col * ld + t] = 0.5 * (y[t] + 0.5 * d[t] * r0 + y[t + 1] - 0.5 * d[t] * r1);
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nk * nw * nmu; e += blockDim.x) {
        const int kw = e / nmu, im = e - kw * nmu, w = kw % nw, col = (kw / nw) * SOLVE_C + w;
        const double *d = C.D + col * ld, *u = C.X + col * ld, *y = C.S + w * ld;
        const double imu = 1.0 / xmu[im];
        double y1 = y[nt - 1], Y = y1;
        for (int k = nt - 2; k >= 0; k--) {
            const double y0 = y[k];
            Y = delo_step(d[k] * imu, Y, y0, y1, u[k]);
            y1 = y0;
        }
        C.I[col * nmu + im] = Y;
    }
}

// LocPrfSph + DeloScalar (solver.f90:182-261) along ray im: opacity x and source y by layer.  One backward
// pass forms each step, derivative and Bezier term where the sweep reaches it; the slopes and reciprocals of a
// point serve its neighbour too.  Grazing rays start from zero intensity at the far side.
__device__ __forceinline__ double sweep_ray(const RayView &R, int im, const double *x, const double *y) {
    const int N = R.n[im];
    const int *mp = R.map + (size_t)im * R.stride;
    const double *dm = R.dm + (size_t)im * R.stride, *idm = R.idm + (size_t)im * R.stride;
    const double *lam = R.lam + (size_t)im * R.stride;
    // TauStep (solver.f90:591-615) from point j to j + 1, given the slope behind (to j + 1) and before
    auto tau = [&](int j, double xb, double xc, double der, double der1) {
        const double yp = j == 0 ? der1 : hmean(der, der1, lam[j]);
        return dm[j] * (xc + 2.0 * xb + dm[j] * 0.5 * yp) * (1.0 / 3.0);
    };
    int l1 = mp[N - 1], l0 = mp[N - 2], lp = N > 2 ? mp[N - 3] : 0;
    double xc = x[l1], xb = x[l0], xa = x[lp];
    double sl1 = (xc - xb) * idm[N - 2], sl0 = N > 2 ? (xb - xa) * idm[N - 3] : 0.0;
    double dcur = tau(N - 2, xb, xc, sl0, sl1), icur = rcp64_step(dcur);
    double y1 = y[l1], y0 = y[l0];
    double g1 = (y1 - y0) * icur, r1 = g1;               // slope of the source over the step; CentDer at j + 1
    double Y = R.graz[im] ? 0.0 : y1;
    for (int j = N - 2; j >= 0; j--) {
        double r0 = g1, dprev = 0.0, iprev = 0.0, g0 = 0.0, yp = 0.0;
        if (j > 0) {                                     // the step from j - 1 to j
            xc = xb; xb = xa;
            if (j > 1) { lp = mp[j - 2]; xa = x[lp]; }
            sl1 = sl0;
            sl0 = j > 1 ? (xb - xa) * idm[j - 2] : 0.0;
            dprev = tau(j - 1, xb, xc, sl0, sl1);
            iprev = rcp64_step(dprev);
            yp = y[mp[j - 1]];
            g0 = (y0 - yp) * iprev;
            r0 = hmean(g0, g1, lambda_of(dprev, dcur));
        }
        const double u = 0.5 * (y0 + 0.5 * dcur * r0 + y1 - 0.5 * dcur * r1);
        Y = delo_step(dcur, Y, y0, y1, u);
        r1 = r0; dcur = dprev; icur = iprev; g1 = g0; y1 = y0; y0 = yp;
    }
    return Y;
}

__device__ __forceinline__ void solve_sph(const Columns &C, int nw, int nk, const RayView &R) {
    const int nmu = R.nmu, ld = C.ld;
    for (int e = threadIdx.x; e < nk * nw * nmu; e += blockDim.x) {
        const int kw = e / nmu, im = e - kw * nmu, w = kw % nw, col = (kw / nw) * SOLVE_C + w;
        C.I[col * nmu + im] = sweep_ray(R, im, C.X + col * ld, C.S + w * ld);
    }
}

// RadTranCalc + disk integration; R.nmu > 0: along the rays of a spherical model.  Without spl and sfl only
// the continuum is solved (as MagRadTranCalc needs).
template <bool SPH>
__device__ __forceinline__ void radtran_cta(const AtmView &A, const double *__restrict__ lineopac,
                                            const double *__restrict__ rhox, int nmu, const double *__restrict__ xmu,
                                            const RayView &R, const double *__restrict__ wmu, double *spl, double *spc,
                                            double *sfl, double *sfc) {
    extern __shared__ double sm[];
    __shared__ double c1_s[SOLVE_C], c2_s[SOLVE_C];
    const int nt = A.ntau, w0 = blockIdx.x * SOLVE_C, nw = min(SOLVE_C, A.nwl - w0);
    const int nk = (spl || sfl) ? 2 : 1;                 // kinds computed: 0 continuum, 1 line
    const Columns C = columns(sm, nt, nmu);
    if (threadIdx.x < nw) {
        const double wl = A.wave[w0 + threadIdx.x] + A.wfirst;
        c1_s[threadIdx.x] = FSG_HC * FSG_VC * 1e13 / FSG_KBOLT / wl;
        c2_s[threadIdx.x] = exp(50.7649141 - 5.0 * log(wl));
    }
    __syncthreads();
    for (int e = threadIdx.x; e < nw * nt; e += blockDim.x) {
        const int w = e / nt, t = e - w * nt;
        const size_t g = (size_t)w0 * nt + e;
        const double c = A.contopac[g];
        C.X[w * C.ld + t] = c;
        if (nk == 2) C.X[(SOLVE_C + w) * C.ld + t] = c + lineopac[g];
        C.S[w * C.ld + t] = planck(c1_s[w], c2_s[w], A.xi[XI_T * nt + t]);
    }
    __syncthreads();
    if (SPH) solve_sph(C, nw, nk, R);
    else solve_pp(C, nt, nw, nk, nmu, rhox, xmu);
    __syncthreads();
    for (int e = threadIdx.x; e < nk * nw * nmu; e += blockDim.x) {
        const int kind = e / (nw * nmu), r = e - kind * nw * nmu;
        double *out = kind == 0 ? spc : spl;
        if (out) out[(size_t)w0 * nmu + r] = C.I[kind * SOLVE_C * nmu + r];
    }
    // disk integration without broadening: Sf = sum over mu of Sp * Wmu (convol.f90:233-234)
    for (int e = threadIdx.x; e < nk * nw; e += blockDim.x) {
        const int kind = e / nw, w = e - kind * nw;
        double a = 0.0;
        for (int im = 0; im < nmu; im++) a = a + C.I[(kind * SOLVE_C + w) * nmu + im] * wmu[im];
        double *out = kind == 0 ? sfc : sfl;
        if (out) out[w0 + w] = a;
    }
}

__global__ void k_radtran(AtmView A, const double *__restrict__ lineopac, const double *__restrict__ rhox, int nmu,
                          const double *__restrict__ xmu, const double *__restrict__ wmu, double *spl, double *spc,
                          double *sfl, double *sfc) {
    radtran_cta<false>(A, lineopac, rhox, nmu, xmu, RayView{}, wmu, spl, spc, sfl, sfc);
}

__global__ void k_radtran_sph(AtmView A, const double *__restrict__ lineopac, RayView R,
                              const double *__restrict__ wmu, double *spl, double *spc, double *sfl, double *sfc) {
    radtran_cta<true>(A, lineopac, nullptr, R.nmu, nullptr, R, wmu, spl, spc, sfl, sfc);
}

int fsg_launch_radtran(cudaStream_t s, const AtmView &A, const double *lineopac, const double *rhox, int nmu,
                       const double *xmu, const double *wmu, double *spl, double *spc, double *sfl, double *sfc) {
    k_radtran<<<(A.nwl + SOLVE_C - 1) / SOLVE_C, columns_threads(nmu), columns_smem(A.ntau, nmu), s>>>(
        A, lineopac, rhox, nmu, xmu, wmu, spl, spc, sfl, sfc);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

int fsg_launch_radtran_sph(cudaStream_t s, const AtmView &A, const double *lineopac, const RayView &R,
                           const double *wmu, double *spl, double *spc, double *sfl, double *sfc) {
    k_radtran_sph<<<(A.nwl + SOLVE_C - 1) / SOLVE_C, columns_threads(R.nmu), columns_smem(A.ntau, R.nmu), s>>>(
        A, lineopac, R, wmu, spl, spc, sfl, sfc);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

// LinStrCalc (synth.f90:1774-1822): central depth of each retained line from the continuum and continuum +
// line intensities at its centre (the centre opacities of the central pass: ContOpac at Wlcent, LineOpacity2
// at Wlcent), disk-integrated with Wmu when nmu > 1; 0 for rejected lines.  The columns of a CTA are the
// centres of SOLVE_C lines.
__global__ void k_linstr(AtmView A, LineView L, const float *__restrict__ vtab, const double *__restrict__ anode,
                         const double *__restrict__ aida, const int32_t *__restrict__ flags, int nmu,
                         const double *__restrict__ xmu, const double *__restrict__ wmu,
                         const double *__restrict__ rhox, RayView R, float *linstr) {
    extern __shared__ double sm[];
    __shared__ XCoef xc_s[SOLVE_C];
    __shared__ double c1_s[SOLVE_C], c2_s[SOLVE_C], dw_s[SOLVE_C];
    __shared__ int iwl_s[SOLVE_C], keep_s[SOLVE_C];
    const int nt = A.ntau;
    const int64_t i0 = (int64_t)blockIdx.x * SOLVE_C;
    const int nw = (int)(L.n - i0 < SOLVE_C ? L.n - i0 : SOLVE_C);
    const Columns C = columns(sm, nt, nmu);
    int any = 0;
    if (threadIdx.x < nw) {
        const int64_t i = i0 + threadIdx.x;
        const int keep = !(flags[i] & FSG_F_WEAK);
        keep_s[threadIdx.x] = keep;
        any = keep;
        if (keep) {
            const double wlc = L.wl[i] - A.wfirst, wl = wlc + A.wfirst;
            xline_setup(A, L, i, wlc, line_input_flags(L, i, 0), &xc_s[threadIdx.x]);
            const int iwl = waveidx(A, wlc);
            iwl_s[threadIdx.x] = iwl;
            dw_s[threadIdx.x] = (wlc - A.wave[iwl - 1]) / (A.wave[iwl] - A.wave[iwl - 1]);
            c1_s[threadIdx.x] = FSG_HC * FSG_VC * 1e13 / FSG_KBOLT / wl;
            c2_s[threadIdx.x] = exp(50.7649141 - 5.0 * log(wl));
        }
    }
    if (!__syncthreads_or(any)) {
        if (threadIdx.x < nw) linstr[i0 + threadIdx.x] = 0.0f;
        return;
    }
    for (int e = threadIdx.x; e < nw * nt; e += blockDim.x) {
        const int w = e / nt, t = e - w * nt;
        double co = 1.0, lo = 0.0, src = 1.0;            // rejected lines: a column that is solved and dropped
        if (keep_s[w]) {
            const XCoef &XC = xc_s[w];
            double cop, vv, av;
            xline_depth(A, t, XC, &cop, &vv, &av);
            const double dWl = XC.IxHe > 0 ? 0.0 - A.heshf[(XC.IxHe - 1) * nt + t] : 0.0;
            lo = hvoigt64(vtab, anode, aida, av, dWl * vv) * cop;
            if (A.motype == 1) lo = lo / A.contstd[t];
            co = cont_center(A, iwl_s[w], dw_s[w], t);
            src = planck(c1_s[w], c2_s[w], A.xi[XI_T * nt + t]);
        }
        C.X[w * C.ld + t] = co;
        C.X[(SOLVE_C + w) * C.ld + t] = co + lo;
        C.S[w * C.ld + t] = src;
    }
    __syncthreads();
    if (R.nmu > 0) solve_sph(C, nw, 2, R);               // spherical: LocPrfSph (synth.f90:1801-1803)
    else solve_pp(C, nt, nw, 2, nmu, rhox, xmu);
    __syncthreads();
    if (threadIdx.x >= nw) return;
    const int w = threadIdx.x;
    const double *ic = C.I + w * nmu, *il = C.I + (SOLVE_C + w) * nmu;
    double fl = il[0], fc = ic[0];
    if (nmu > 1) {
        fl = fc = 0.0;
        for (int m = 0; m < nmu; m++) { fl = fl + wmu[m] * il[m]; fc = fc + wmu[m] * ic[m]; }
    }
    linstr[i0 + w] = keep_s[w] ? (float)(1.0 - fl / fc) : 0.0f;
}

void fsg_launch_linstr(cudaStream_t s, const AtmView &A, const LineView &L, const VoigtTables &T,
                       const int32_t *flags, int nmu, const double *xmu, const double *wmu, const double *rhox,
                       const RayView &R, float *linstr) {
    if (L.n > 0)
        k_linstr<<<(unsigned)((L.n + SOLVE_C - 1) / SOLVE_C), columns_threads(nmu), columns_smem(A.ntau, nmu), s>>>(
            A, L, T.vtab, T.anode, T.aida, flags, nmu, xmu, wmu, rhox, R, linstr);
}
