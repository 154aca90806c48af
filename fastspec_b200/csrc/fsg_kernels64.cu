// fsg_kernels64.cu -- FP64 kernels of the line-opacity / formal-solver path (built -fmad=false).
//
//   k_tables        VoigtInit / FVoigtInit (voigt.f90:42-72, 219-251) on the device
//   k_xline_init    XlineInit (opacity.f90:65-93)
//   k_center        LineopCalc central pass (synth.f90:833-907): XlineSetup + XlineDepth,
//                   weak-line bound and centre tests, AnalyticWindow + WaveIdx windows
//   k_params_fast   block refill (synth.f90:1049-1070) into FP32 wing/core records
//   k_params_fp64   block refill into FP64 (LinCop, LinVvgt, LinAvgt) and headers for the plain path
//   k_span          Lstart/Lstop of the plain path's segments (synth.f90:955-978)
//   k_locprf        LocPrfPP over independent profiles (kernel-level entry point; the drivers' solver is in
//                   fsg_solve.cu)
#include "fsg_fp64.cuh"

#include <algorithm>
#include <stdio.h>

// ================================================================================================
// Voigt tables: Chiarella-Reichel (1968) trapezoid sum with pole correction (voigt.f90:158-187,
// 356-393).  Complex arithmetic as gfortran expands it: naive products, Smith's division.
// ================================================================================================
struct cd { double re, im; };
__device__ __forceinline__ cd c_mul(cd a, cd b) {
    double t1 = a.re * b.re, t2 = a.im * b.im, t3 = a.re * b.im, t4 = a.im * b.re;
    return cd{ t1 - t2, t3 + t4 };
}
__device__ __forceinline__ cd c_div(cd a, cd b) {
    double ratio, div, tr, ti;
    if (fabs(b.re) < fabs(b.im)) {
        ratio = b.re / b.im; div = (b.re * ratio) + b.im;
        tr = (a.re * ratio) + a.im; ti = (a.im * ratio) - a.re;
    } else {
        ratio = b.im / b.re; div = (b.im * ratio) + b.re;
        tr = (a.im * ratio) + a.re; ti = a.im - (a.re * ratio);
    }
    return cd{ tr / div, ti / div };
}

__device__ cd cr_sum(double a, double av) {
    const double HH = 0.5;
    cd z{ av, a }, z2 = c_mul(z, z);
    cd s = c_div(cd{ 1.0, 0.0 }, z);
    for (int n = 1; n <= 16; n++) {
        double nh = (double)n * HH;
        double e = exp(-nh * nh);
        cd num{ (2.0 * z.re) * e, (2.0 * z.im) * e };
        cd q = c_div(num, cd{ z2.re - nh * nh, z2.im });
        s.re = s.re + q.re; s.im = s.im + q.im;
    }
    double c = HH / FSG_PI;
    s = cd{ -(c * s.im), c * s.re };
    if (a < 6.0) {
        double p = 2.0 * FSG_PI * a / HH;
        double th = 2.0 * FSG_PI * (2.0 * av - round(2.0 * av));
        double sn = sin(0.5 * th);
        double redd = -(2.0 * exp(0.5 * p) * sinh(0.5 * p)) + exp(p) * 2.0 * (sn * sn);
        double imdd = exp(p) * sin(th);
        double ex = exp(a * a - av * av), ang = -2.0 * a * av;
        cd num{ 2.0 * (ex * cos(ang)), 2.0 * (ex * sin(ang)) };
        cd q = c_div(num, cd{ redd, imdd });
        s.re = s.re + q.re; s.im = s.im + q.im;
    }
    return s;
}

__global__ void k_tables(float *vtab, float2 *fvtab, double *anode, double *aida) {
    const double dv = 8.0 / 1000.0, dt = 2.8284271247461903 / 400.0;
    int iv = blockIdx.x * blockDim.x + threadIdx.x;   // 0..1001
    int ia = blockIdx.y;                              // 0..401
    double aa = ((double)ia * dt) * ((double)ia * dt);
    if (iv == 0) {
        anode[ia] = aa;
        if (ia < FSG_NVA) {
            double an1 = ((double)(ia + 1) * dt) * ((double)(ia + 1) * dt);
            aida[ia] = 1.0 / (an1 - aa);
        } else aida[ia] = 0.0;
    }
    if (iv >= FSG_NV1) return;
    double vv = (double)iv * dv;
    double h, l;
    if (aa <= 0.0) {
        h = exp(-fmin(vv * vv, 700.0));
        int m = 2 * (int)llround(2.0 * vv);
        double x0 = vv - 0.25 * (double)m, p = 0.0;
        for (int n = -31; n <= 31; n += 2) {
            double t = x0 - 0.25 * (double)n;
            p = p + exp(-(t * t)) / (double)(m + n);
        }
        l = (2.0 / FSG_PI) * p;
    } else {
        cd s = cr_sum(aa, vv);
        h = s.re; l = s.im;
    }
    vtab[ia * FSG_NV1 + iv] = (float)h;
    fvtab[ia * FSG_NV1 + iv] = make_float2((float)h, (float)l);
}

// the four VgtTab entries of one bilinear cell side by side
__global__ void k_vtab4(const float *vtab, float4 *vtab4) {
    int iv = blockIdx.x * blockDim.x + threadIdx.x;   // 0..NVV-1
    int r = blockIdx.y;                               // 0..NVA-1
    if (iv >= FSG_NVV) return;
    const float *p0 = vtab + r * FSG_NV1 + iv, *p1 = p0 + FSG_NV1;
    vtab4[r * FSG_NV1 + iv] = make_float4(p0[0], p0[1], p1[0], p1[1]);
}

// (H, L) at two neighbouring v nodes side by side (the last node repeated at the row end)
__global__ void k_fvtab2(const float2 *fvtab, float4 *fvtab2) {
    int iv = blockIdx.x * blockDim.x + threadIdx.x;   // 0..NV1-1
    int r = blockIdx.y;                               // 0..NA1-1
    if (iv >= FSG_NV1) return;
    const float2 a = fvtab[r * FSG_NV1 + iv], b = fvtab[r * FSG_NV1 + min(iv + 1, FSG_NV1 - 1)];
    fvtab2[r * FSG_NV1 + iv] = make_float4(a.x, a.y, b.x, b.y);
}

int fsg_build_tables(VoigtTables *t, cudaStream_t s, std::string *err) {
    cudaError_t e;
    if ((e = cudaMalloc(&t->vtab4, sizeof(float4) * FSG_NVA * FSG_NV1)) != cudaSuccess ||
        (e = cudaMalloc(&t->vtab, sizeof(float) * FSG_NA1 * FSG_NV1)) != cudaSuccess ||
        (e = cudaMalloc(&t->fvtab, sizeof(float2) * FSG_NA1 * FSG_NV1)) != cudaSuccess ||
        (e = cudaMalloc(&t->fvtab2, sizeof(float4) * FSG_NA1 * FSG_NV1)) != cudaSuccess ||
        (e = cudaMalloc(&t->anode, sizeof(double) * FSG_NA1)) != cudaSuccess ||
        (e = cudaMalloc(&t->aida, sizeof(double) * FSG_NA1)) != cudaSuccess) {
        *err = fsg_cuda_msg(e, "table allocation");
        return FSG_E_NOMEM;
    }
    dim3 grid((FSG_NV1 + 127) / 128, FSG_NA1);
    k_tables<<<grid, 128, 0, s>>>(t->vtab, t->fvtab, t->anode, t->aida);
    if ((e = cudaGetLastError()) != cudaSuccess) { *err = fsg_cuda_msg(e, "k_tables"); return FSG_E_CUDA; }
    k_vtab4<<<dim3((FSG_NVV + 127) / 128, FSG_NVA), 128, 0, s>>>(t->vtab, t->vtab4);
    if ((e = cudaGetLastError()) != cudaSuccess) { *err = fsg_cuda_msg(e, "k_vtab4"); return FSG_E_CUDA; }
    k_fvtab2<<<dim3((FSG_NV1 + 127) / 128, FSG_NA1), 128, 0, s>>>(t->fvtab, t->fvtab2);
    if ((e = cudaGetLastError()) != cudaSuccess) { *err = fsg_cuda_msg(e, "k_fvtab2"); return FSG_E_CUDA; }
    return FSG_OK;
}

void fsg_free_tables(VoigtTables *t) {
    cudaFree(t->vtab); cudaFree(t->vtab4); cudaFree(t->fvtab); cudaFree(t->fvtab2); cudaFree(t->anode); cudaFree(t->aida);
    t->vtab = nullptr; t->vtab4 = nullptr; t->fvtab = nullptr; t->fvtab2 = nullptr; t->anode = nullptr; t->aida = nullptr;
}

// ================================================================================================
// XlineInit (opacity.f90:65-93): rows of A.xi
// ================================================================================================
__global__ void k_xline_init(int nt, const double *T, const double *xne, const double *rho,
                             const float *h1, const float *he1, const float *h2, double h2brd,
                             double *xi) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= nt) return;
    double Temp = T[t], Xne = xne[t];
    double Vh = sqrt(2.0 * FSG_KBOLT * Temp / FSG_MH);
    double np = (double)h1[t] + 0.412265 * (double)he1[t];
    if (h2brd > 0.0) np = np + h2brd * 0.874307 * (double)h2[t];
    const double erg2ev = 1e-7 / 1.602176634e-19;
    xi[XI_NPRTB * nt + t] = np;
    xi[XI_GVWPRT * nt + t] = 17.0 * pow(Vh, 0.6) * np;
    xi[XI_TEMP6 * nt + t] = pow(Temp / 1e4, 1.0 / 6.0) * Xne;
    xi[XI_TEMP3 * nt + t] = pow(Temp / 1e4, 0.3) * np;
    xi[XI_KBT * nt + t] = FSG_KBOLT * Temp;
    xi[XI_KBET * nt + t] = FSG_KBOLT * erg2ev * Temp;
    xi[XI_T * nt + t] = Temp;
    xi[XI_XNE * nt + t] = Xne;
    xi[XI_RHO * nt + t] = rho[t];
}

void fsg_launch_xline_init(cudaStream_t s, int nt, const double *T, const double *xne, const double *rho,
                           const float *h1, const float *he1, const float *h2, double h2brd, double *xi) {
    k_xline_init<<<(nt + 127) / 128, 128, 0, s>>>(nt, T, xne, rho, h1, he1, h2, h2brd, xi);
}

// ================================================================================================
// Central pass (synth.f90:833-907).  One sweep over depth: XlineDepth once per
// depth feeds the LinCop bound test against the continuum, the single-line opacity at the line centre
// (LineOpacity2) and AnalyticWindow; no Ntau-long arrays are held.
// ================================================================================================
__device__ __forceinline__ double center_shift(const AtmView &A, int ihe, int t) {
    return (ihe > 0) ? A.heshf[(ihe - 1) * A.ntau + t] : 0.0;
}

// The per-line part before the sweep and one depth of the three maxima the reference takes in turn
// (synth.f90:876-907): (1) the upper bound LinCop / ContOpac (H(a, v) <= 1), (2) the single-line opacity at
// the line centre (LineOpacity2 at Wl = Wlcent) and (3) the AnalyticWindow half-width (opacity.f90:678-710).
// Each is a maximum over depths of per-depth values that do not depend on the others, so computing
// XlineDepth once per depth for all three gives the reference's tests and windows exactly; the
// later maxima are used only when the earlier tests keep the line.
struct CenterLine { XCoef XC; double wlc, dW; int f, iwl; };
__device__ __forceinline__ CenterLine center_line(const AtmView &A, const LineView &L, int64_t i) {
    CenterLine c;
    c.f = line_input_flags(L, i, 0);
    c.wlc = L.wl[i] - A.wfirst;
    xline_setup(A, L, i, c.wlc, c.f, &c.XC);
    if (c.XC.IxHe > 0) c.f |= (c.XC.IxHe << 8);
    c.iwl = waveidx(A, c.wlc);
    c.dW = (c.wlc - A.wave[c.iwl - 1]) / (A.wave[c.iwl] - A.wave[c.iwl - 1]);
    return c;
}
__device__ __forceinline__ void center_depth(const AtmView &A, const CenterLine &c, int t, const float *__restrict__ vtab,
                                             const double *__restrict__ anode, const double *__restrict__ aida,
                                             double &mx1, double &mx2, double &dWwin) {
    const double iSqrtPi = 0.5641895835477563;
    const int ihe = c.XC.IxHe;
    double cop, vv, av;
    xline_depth(A, t, c.XC, &cop, &vv, &av);
    const double co = cont_center(A, c.iwl, c.dW, t);
    mx1 = fmax(mx1, (A.motype == 1) ? cop / (co * A.contstd[t]) : cop / co);
    double dWl = 0.0;
    if (ihe > 0) dWl = 0.0 - center_shift(A, ihe, t);
    double lo = hvoigt64(vtab, anode, aida, av, dWl * vv) * cop;
    if (A.motype == 1) lo = lo / A.contstd[t];
    mx2 = fmax(mx2, lo / co);
    double r = cop / (A.epsopac * co);
    if (A.motype == 1) r = r / A.contstd[t];
    if (r <= 1.0) return;
    double w = sqrt(log(r) + fmax(0.0, av * (r * iSqrtPi - av))) / vv;
    if (ihe > 0) w = w + fabs(center_shift(A, ihe, t));
    dWwin = fmax(dWwin, w);
}
// flags and window of the line from the maxima; whether it is kept
__device__ __forceinline__ bool center_result(const AtmView &A, const CenterLine &c, double mx1, double mx2, double dWwin,
                                              int64_t i, int32_t *flags, int32_t *ileft, int32_t *iright) {
    int f = c.f, il = 1, ir = A.nwl;
    if (mx1 < A.epsopac || mx2 < A.epsopac) {
        f |= FSG_F_WEAK;
    } else {
        il = waveidx(A, c.wlc - dWwin);                    // WaveIdx (synth.f90:904-906)
        ir = waveidx(A, c.wlc + dWwin) + 1;
        if (ir > A.nwl) ir = A.nwl;
    }
    flags[i] = f; ileft[i] = il; iright[i] = ir;
    return !(f & FSG_F_WEAK);
}

// One thread per line.  Eight 128-thread CTAs per SM (64 registers, a few spilled): the sweep is bound by the
// FP64 pipe, and the extra resident warps hide more of its latency (177 -> 150 ms on the 1e8-line list).
__global__ void __launch_bounds__(128, 8) k_center(AtmView A, LineView L, const float *__restrict__ vtab,
                         const double *__restrict__ anode, const double *__restrict__ aida,
                         int32_t *flags, int32_t *ileft, int32_t *iright, unsigned long long *nkeep) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= L.n) return;
    const CenterLine c = center_line(A, L, i);
    double mx1 = -1.0e308, mx2 = -1.0e308, dWwin = 0.0;
    for (int t = 0; t < A.ntau; t++) center_depth(A, c, t, vtab, anode, aida, mx1, mx2, dWwin);
    const bool keep = center_result(A, c, mx1, mx2, dWwin, i, flags, ileft, iright);
    // warp-aggregated count of retained lines
    unsigned m = __ballot_sync(__activemask(), keep);
    if ((threadIdx.x & 31) == (__ffs(__activemask()) - 1) && m) atomicAdd(nkeep, (unsigned long long)__popc(m));
}

// One warp per line, lanes over depths: the same values, and maxima are exact in any order.
__global__ void __launch_bounds__(128) k_center_warp(AtmView A, LineView L, const float *__restrict__ vtab,
                         const double *__restrict__ anode, const double *__restrict__ aida,
                         int32_t *flags, int32_t *ileft, int32_t *iright, unsigned long long *nkeep) {
    const int64_t i = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (i >= L.n) return;                                // whole warps leave together
    const CenterLine c = center_line(A, L, i);
    double mx1 = -1.0e308, mx2 = -1.0e308, dWwin = 0.0;
    for (int t = lane; t < A.ntau; t += 32) center_depth(A, c, t, vtab, anode, aida, mx1, mx2, dWwin);
    for (int o = 16; o > 0; o >>= 1) {
        mx1 = fmax(mx1, __shfl_xor_sync(0xffffffffu, mx1, o));
        mx2 = fmax(mx2, __shfl_xor_sync(0xffffffffu, mx2, o));
        dWwin = fmax(dWwin, __shfl_xor_sync(0xffffffffu, dWwin, o));
    }
    if (lane == 0 && center_result(A, c, mx1, mx2, dWwin, i, flags, ileft, iright)) atomicAdd(nkeep, 1ull);
}

// A thread's sweep over the depths takes 2.3 us a depth whatever the number of lines (the latency of an FP64 chain), and
// a list fills the GPU with threads from 150,000 lines on; a warp per line repeats the line's set-up in every
// lane, 1.7 us more per thousand lines up to 32 depths, 2.7 up to 64, 3.7 up to 96.  56 depths, with the call's own 25 us:
// 300 lines 140 us by threads, 32 us by warps; 20,000: 144 and 81 us.  The two meet near 8,000 lines at 8 depths (42 and
// 45 us), 20,000 at 20 (69 us), 31,000 at 33 (105 us).
void fsg_launch_center(cudaStream_t s, const AtmView &A, const LineView &L, const VoigtTables &T,
                       int32_t *flags, int32_t *ileft, int32_t *iright, unsigned long long *nkeep) {
    if (L.n <= 0) return;
    if (L.n <= std::min(32768, 950 * A.ntau))
        k_center_warp<<<(unsigned)((L.n + 3) / 4), 128, 0, s>>>(A, L, T.vtab, T.anode, T.aida, flags, ileft, iright, nkeep);
    else
        k_center<<<(unsigned)((L.n + 127) / 128), 128, 0, s>>>(A, L, T.vtab, T.anode, T.aida, flags, ileft, iright, nkeep);
}

// ================================================================================================
// Block refill: per retained line of the block, XlineSetup once then XlineDepth over depths.
// ================================================================================================

// Line j of the block is list line idx[j0 + j * stride].  One warp per group of lpw lines (32, fewer where
// the lines are too few to fill the GPU with such groups): lane k runs XlineSetup for line k of the group
// into shared memory, then the warp walks the group's (line, depth) pairs in record order, one pair per
// lane, so that each store of wing and core records covers consecutive records of the arrays; depths are
// padded to an even count, so that neighbouring lanes hold the two halves of a wing pair.  The per-line
// maximum core half-width and the minimum vv2 are reduced over each line's run of lanes with shuffles (a
// run is a line's depths in one step) and merged into shared memory by the run's first lane; lane k then
// writes the header of line k.  Both reductions are exact (max / min), so the records and headers do not
// depend on the order in which depths are taken.
#define PF_WARPS 4
__global__ void __launch_bounds__(PF_WARPS * 32)
k_params_fast(AtmView A, LineView L, const int64_t *__restrict__ idx, int64_t j0, int64_t stride,
              int64_t nb, int lpw, const int32_t *__restrict__ flags,
              const int32_t *__restrict__ ileft, const int32_t *__restrict__ iright,
              const double *__restrict__ anode, const double *__restrict__ aida,
              WingPair *wing, CoreRec *core, LineHdr *hdr) {
    __shared__ XCoef xs[PF_WARPS][32];
    __shared__ unsigned long long hcs[PF_WARPS][32];   // bits of hcore + 1 (0: no depth has a core)
    __shared__ unsigned vms[PF_WARPS][32];             // bits of the smallest vv2 (non-negative floats)
    __shared__ double xms[PF_WARPS][32];               // largest dl^2 in the window
    __shared__ int big[PF_WARPS][32];                  // some depth leaves the range of paired denominators
    const int wp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t jb = ((int64_t)blockIdx.x * PF_WARPS + wp) * lpw;
    if (jb >= nb) return;                               // whole warps only: no block barrier below
    const int ng = (nb - jb < lpw) ? (int)(nb - jb) : lpw;
    const int nt = A.ntau, ntp = 2 * wing_pairs(nt);
    int64_t i = 0; int f = 0; double wlc = 0.0;
    if (lane < ng) {
        i = idx[j0 + (jb + lane) * stride];
        f = flags[i];
        wlc = L.wl[i] - A.wfirst;
        xline_setup(A, L, i, wlc, f, &xs[wp][lane]);
        const int il = max(ileft[i], 1), ir = min(iright[i], A.nwl);
        double xm = 0.0;
        if (il <= ir) {
            const double dl = wlc - A.wave[il - 1], dr = wlc - A.wave[ir - 1];
            xm = fmax(dl * dl, dr * dr);
        }
        xms[wp][lane] = xm;
    }
    big[wp][lane] = 0;
    hcs[wp][lane] = 0ull;
    vms[wp][lane] = __float_as_uint(3.0e38f);
    __syncwarp();
    const int tot = ng * ntp;
    float4 *wg = (float4 *)(wing + (size_t)jb * wing_pairs(nt));      // half q of the group's pairs: depth q of the walk
    CoreRec *cg = core + (size_t)jb * nt;
    // pair p = lane + step: line ln = p / ntp, depth t = p % ntp, advanced by 32 per step
    int ln = lane / ntp, t = lane - (lane / ntp) * ntp;
    for (int p0 = 0; p0 < tot; p0 += 32) {
        const int p = p0 + lane;
        const bool on = p < tot;
        double hc = -1.0;          // this pair's core half-width (s < 196), -1 when none
        float vv2 = 3.0e38f;
        float wv2 = 0.0f, c2m1 = 0.0f, twoA = 0.0f, c1 = 0.0f;
        if (on && t < nt) {
            const XCoef &XC = xs[wp][ln];
            double cop, vv, av;
            xline_depth(A, t, XC, &cop, &vv, &av);
            if (A.motype == 1) cop = cop / A.contstd[t];     // LineOpacity1 divides the sum by ContOpacStd
            double a2 = av * av;
            wv2 = (float)(vv * vv);
            c2m1 = (float)(a2 - 0.5);
            twoA = (float)(2.0 * a2);
            c1 = (float)(cop * av * FSG_SQRTPIINV);
            vv2 = wv2;
            if (!(xms[wp][ln] * wv2 + a2 < 2147483648.0 && fabsf(c1) < 1073741824.0f)) big[wp][ln] = 1;
            CoreRec c;
            c.vv = vv; c.cop = (float)cop; c.a = (float)av; c.vv2 = wv2; c.c2m1 = c2m1;
            // table row and weight of a in FP64 (sqrt(a) nodes, voigt.f90:84-92); ia = 0: a >= 8
            if (!(av < 8.0)) { c.ia = 0; c.ua = 0.0f; }
            else if (av < anode[1]) { c.ia = 1; c.ua = (float)(av * aida[0]); }
            else {
                const int ia = min((int)(sqrt(av) * (1.0 / (2.8284271247461903 / 400.0))) + 1, FSG_NVA);
                c.ia = ia;
                c.ua = (float)((av - anode[ia - 1]) * aida[ia - 1]);
            }
            cg[(size_t)ln * nt + t] = c;
            // the accumulation evaluates the core form where fl32(dl^2 vv2 + c2m1) < 195.5; a margin
            // of 0.05 in s and 1e-5 in dl covers the FP32 rounding of the records and of dl^2
            double q = 196.05 - a2;
            if (q > 0.0) hc = sqrt(q) / vv * (1.0 + 1e-5);
        }
        // the two depths of a wing pair sit in neighbouring lanes: the even one stores (vv2, c2m1) of
        // both, the odd one (twoA, c1)
        {
            const bool odd = lane & 1;
            const float s0 = odd ? wv2 : twoA, s1 = odd ? c2m1 : c1;
            const float r0 = __shfl_xor_sync(0xffffffffu, s0, 1), r1 = __shfl_xor_sync(0xffffffffu, s1, 1);
            if (on) wg[p] = odd ? make_float4(r0, twoA, r1, c1) : make_float4(wv2, r0, c2m1, r1);
        }
        // segmented reduction over the run of lanes that share this lane's line (lanes past the
        // last pair form their own run at the end); the run's first lane ends with the run's value
        #pragma unroll
        for (int off = 1; off < 32; off <<= 1) {
            double oh = __shfl_down_sync(0xffffffffu, hc, off);
            float ov = __shfl_down_sync(0xffffffffu, vv2, off);
            if (lane + off < 32 && t + off < ntp) { hc = fmax(hc, oh); vv2 = fminf(vv2, ov); }
        }
        if (on && (lane == 0 || t == 0)) {
            if (hc >= 0.0) atomicMax(&hcs[wp][ln], (unsigned long long)__double_as_longlong(hc) + 1ull);
            atomicMin(&vms[wp][ln], __float_as_uint(vv2));
        }
        t += 32;
        while (t >= ntp) { t -= ntp; ln++; }
    }
    __syncwarp();
    if (lane >= ng) return;
    const unsigned long long hb = hcs[wp][lane];
    const double hcore = hb ? __longlong_as_double((long long)(hb - 1ull)) : -1.0;
    const float vv2min = __uint_as_float(vms[wp][lane]);
    LineHdr h;
    h.wlh = (float)wlc;
    h.wll = (float)(wlc - (double)h.wlh);
    h.ileft = max(ileft[i], 1); h.iright = min(iright[i], A.nwl);       // given windows may reach past the grid
    h.cl = 1; h.cr = 0;
    if (f & FSG_F_WEAK) { h.ileft = 1; h.iright = 0; }    // rejected line (batched lists): empty window
    else if (hcore >= 0.0) {
        // 1-based indices of the first wavelength >= wlc - hcore and the last <= wlc + hcore,
        // widened by one wavelength and clipped to the window
        int a = lower_index(A.wave, A.nwl, wlc - hcore) + 1;
        int b = lower_index(A.wave, A.nwl, wlc + hcore);
        if (b < A.nwl && A.wave[b] == wlc + hcore) b++;
        int cl = max(a - 1, h.ileft), cr = min(b + 1, h.iright);
        if (cl <= cr) { h.cl = cl; h.cr = cr; }
    }
    // pairable: the line may share a reciprocal in the wing pass (no depth's denominator above 2^62, no coefficient
    // above 2^30: the product of two stays below 2^126, its numerator finite)
    // x offset that silences a point in the wing pass: with dl^2 replaced by 1e19 / min vv2, every
    // depth has t >= 1e19, so t^2 >= 1e38 and the FP32 reciprocal (flush-to-zero) is exactly 0 while
    // c1 (t + 1) stays finite; the point then adds exactly 0
    h.silent = __float_as_int(1.0e19f / vv2min);
    h.pairable = !big[wp][lane];
    hdr[jb + lane] = h;
}

void fsg_launch_params_fast(cudaStream_t s, const AtmView &A, const LineView &L, const int64_t *idx,
                            int64_t j0, int64_t stride, int64_t nb, const int32_t *flags, const int32_t *ileft,
                            const int32_t *iright, const VoigtTables &T, WingPair *wing, CoreRec *core,
                            LineHdr *hdr) {
    if (nb <= 0) return;
    // 32 lines per warp once that gives every SM 16 warps (75,776 lines); below, as many warps of fewer lines
    const int64_t warps = 148 * 16;
    const int lpw = (int)std::min<int64_t>(32, (nb + warps - 1) / warps);
    const int64_t per = (int64_t)PF_WARPS * lpw;
    k_params_fast<<<(unsigned)((nb + per - 1) / per), PF_WARPS * 32, 0, s>>>(A, L, idx, j0, stride, nb, lpw, flags, ileft,
                                                                            iright, T.anode, T.aida, wing, core, hdr);
}

// FP64 records of the plain path: row q holds the list line list[q] (list null: i0 + q) as
// p64[q][t] = (LinCop, LinVvgt, LinAvgt) and its header.  Lines with any flag of skip get an empty
// window.  Magnetic lists give their Zeeman components (Z, line i's at zmap[i]): the core range is widened
// by the largest component shift, and the header keeps zmap[i].  One warp per line, lanes over depths: XlineDepth's FP64 chain is long, and a thread per line
// walked all depths one after another (84 + 71 us for the 19,362 lines of a 200 A solar list, narrow and wide).
__global__ void __launch_bounds__(128)
k_params_fp64(AtmView A, LineView L, const int64_t *__restrict__ list, int64_t i0, int64_t nb, int skip,
              const int32_t *__restrict__ flags, const int32_t *__restrict__ ileft,
              const int32_t *__restrict__ iright, ZView Z, const int64_t *__restrict__ zmap, double3 *p64,
              LineHdr64 *hdr) {
    const int64_t q = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (q >= nb) return;                                // whole warps leave together
    const int64_t i = list ? list[q] : i0 + q;
    const int f = flags[i], nt = A.ntau;
    LineHdr64 h;
    h.wlc = L.wl[i] - A.wfirst;
    h.il = 1; h.ir = 0; h.cl = 1; h.cr = 0; h.ihe = (f >> 8) & 255; h.zi = zmap ? (int)zmap[i] : 0;
    if (f & skip) { if (lane == 0) hdr[q] = h; return; }
    XCoef XC;
    xline_setup(A, L, i, h.wlc, f, &XC);
    double hcore = -1.0, shmax = 0.0;
    for (int t = lane; t < nt; t += 32) {
        double cop, vv, av;
        xline_depth(A, t, XC, &cop, &vv, &av);
        p64[(size_t)q * nt + t] = make_double3(cop, vv, av);
        const double r = 196.05 - av * av;
        if (r > 0.0) hcore = fmax(hcore, sqrt(r) / vv * (1.0 + 1e-5));
        if (h.ihe > 0) shmax = fmax(shmax, fabs(A.heshf[(size_t)(h.ihe - 1) * nt + t]));
    }
    if (zmap) {
        double zmax = 0.0;
        for (int k = lane; k < Z.npi[h.zi]; k += 32) zmax = fmax(zmax, fabs((double)Z.splpi[Z.pi_off[h.zi] + k]));
        for (int k = lane; k < Z.nsi[h.zi]; k += 32) zmax = fmax(zmax, fabs((double)Z.splsi[Z.si_off[h.zi] + k]));
        for (int o = 16; o > 0; o >>= 1) zmax = fmax(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
        shmax += zmax;
    }
    for (int o = 16; o > 0; o >>= 1) {
        hcore = fmax(hcore, __shfl_xor_sync(0xffffffffu, hcore, o));
        shmax = fmax(shmax, __shfl_xor_sync(0xffffffffu, shmax, o));
    }
    if (lane != 0) return;
    h.il = ileft[i]; h.ir = iright[i];
    if (hcore >= 0.0) {
        // 1-based indices of the first wavelength >= wlc - half and the last <= wlc + half, widened by one
        // and clipped to the window
        const double half = hcore + shmax;
        int a = lower_index(A.wave, A.nwl, h.wlc - half) + 1;
        int b = lower_index(A.wave, A.nwl, h.wlc + half);
        if (b < A.nwl && A.wave[b] == h.wlc + half) b++;
        const int cl = max(a - 1, h.il), cr = min(b + 1, h.ir);
        if (cl <= cr) { h.cl = cl; h.cr = cr; }
    }
    hdr[q] = h;
}

void fsg_launch_params_fp64(cudaStream_t s, const AtmView &A, const LineView &L, const int64_t *list, int64_t i0,
                            int64_t nb, int skip, const int32_t *flags, const int32_t *il, const int32_t *ir,
                            const ZView *Z, const int64_t *zmap, double3 *p64, LineHdr64 *hdr) {
    if (nb <= 0) return;
    k_params_fp64<<<(unsigned)((nb + 3) / 4), 128, 0, s>>>(A, L, list, i0, nb, skip, flags, il, ir, Z ? *Z : ZView{},
                                                          Z ? zmap : nullptr, p64, hdr);
}

// ================================================================================================
// Plain FP64 path: Lstart/Lstop pointers (synth.f90:955-978); the sums are in fsg_accum64.cu.
// ================================================================================================
__global__ void k_span(int64_t n, const int32_t *flags, const int32_t *ileft, const int32_t *iright,
                       int *lstart, int *lstop) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int f = flags[i];
    if ((f & FSG_F_WEAK) || (f & FSG_F_WIDE)) return;
    for (int w = ileft[i]; w <= iright[i]; w++) {
        atomicMin(&lstart[w - 1], (int)(i + 1));
        atomicMax(&lstop[w - 1], (int)(i + 1));
    }
}

void fsg_launch_span(cudaStream_t s, int64_t n, const int32_t *flags, const int32_t *ileft,
                     const int32_t *iright, int *lstart, int *lstop) {
    if (n <= 0) return;
    k_span<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(n, flags, ileft, iright, lstart, lstop);
}

// ================================================================================================
// Elemental HVoigt / FVoigt over arrays (kernel-level entry points)
// ================================================================================================
__global__ void k_hvoigt(int64_t n, const double *a, const double *v, double *h, const float *vtab,
                         const double *anode, const double *aida) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) h[i] = hvoigt64(vtab, anode, aida, a[i], v[i]);
}

__global__ void k_fvoigt(int64_t n, const double *a, const double *v, double *h, double *l,
                         const float2 *fvtab, const double *anode, const double *aida) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    // FVoigt (voigt.f90:256-299): same a-state rule as HVoigt
    double A = a[i], V = v[i], av = fabs(V), vg, fv;
    if (A < 8.0 && av < 8.0) {
        VLine64 L;
        L.A = A;
        if (A < anode[1]) { L.IA = 1; L.UA = A * aida[0]; }
        else { L = vline64(anode, aida, A); }
        fvoigt_line64(fvtab, L, V, &vg, &fv);
    } else { fv_asym64(A, av, &vg, &fv); fv = copysign(fabs(fv), V); }
    h[i] = vg; l[i] = fv;
}

void fsg_launch_hvoigt(cudaStream_t s, int64_t n, const double *a, const double *v, double *h,
                       const VoigtTables &T) {
    if (n > 0) k_hvoigt<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, a, v, h, T.vtab, T.anode, T.aida);
}
void fsg_launch_fvoigt(cudaStream_t s, int64_t n, const double *a, const double *v, double *h, double *l,
                       const VoigtTables &T) {
    if (n > 0) k_fvoigt<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, a, v, h, l, T.fvtab, T.anode, T.aida);
}

// LocPrfPP over independent profiles: one thread per profile (kernel-level entry point)
// LocPrfPP (solver.f90:123-179) of one profile: x = Xki, y = Src over nt depths, d/r/u work arrays
// of nt doubles each; the nmu emergent intensities go to out[0 .. nmu-1]
__device__ void locprf_one(int nmu, const double *xmu, int nt, const double *x, const double *y,
                           const double *rhox, double *d, double *r, double *u, double *out) {
    // TauStep
    {
        double Dx1 = (rhox[1] - rhox[0]) / 1.0, Yp = (x[1] - x[0]) / Dx1;
        d[0] = Dx1 * (x[1] + 2.0 * x[0] + Dx1 / 2.0 * Yp) / 3.0;
        for (int k = 2; k <= nt - 1; k++) {
            double Dx = (rhox[k - 1] - rhox[k - 2]) / 1.0; Dx1 = (rhox[k] - rhox[k - 1]) / 1.0;
            double Der = (x[k - 1] - x[k - 2]) / Dx, Der1 = (x[k] - x[k - 1]) / Dx1;
            if (Der * Der1 > 0.0) {
                double Lambda = (1.0 + Dx1 / (Dx + Dx1)) / 3.0;
                Yp = (Der / (Lambda * Der1 + (1.0 - Lambda) * Der)) * Der1;
            } else Yp = 0.0;
            d[k - 1] = Dx1 * (x[k] + 2.0 * x[k - 1] + Dx1 / 2.0 * Yp) / 3.0;
        }
    }
    for (int k = 2; k <= nt - 1; k++) {
        double Dx = d[k - 2], Dx1 = d[k - 1];
        double InvDx = 1.0 / Dx, InvDx1 = 1.0 / Dx1;
        double Lambda = (1.0 + Dx1 / (Dx + Dx1)) / 3.0, Lambda1 = 1.0 - Lambda;
        double Der = (y[k - 1] - y[k - 2]) * InvDx, Der1 = (y[k] - y[k - 1]) * InvDx1;
        r[k - 1] = (Der * Der1 > 0.0) ? (Der / (Lambda * Der1 + Lambda1 * Der)) * Der1 : 0.0;
    }
    r[0] = (y[1] - y[0]) / d[0];
    r[nt - 1] = (y[nt - 1] - y[nt - 2]) / d[nt - 2];
    for (int k = 0; k < nt - 1; k++) u[k] = 0.5 * (y[k] + 0.5 * d[k] * r[k] + y[k + 1] - 0.5 * d[k] * r[k + 1]);
    for (int im = 0; im < nmu; im++) {
        double Imu = 1.0 / xmu[im], Y = y[nt - 1];
        for (int k = nt - 2; k >= 0; k--) {
            double Eps, Alpha, Beta, Gamma;
            delo_coef(d[k] * Imu, Eps, Alpha, Beta, Gamma);
            Y = Y * Eps + Alpha * y[k] + Beta * y[k + 1] + Gamma * u[k];
        }
        out[im] = Y;
    }
}

__global__ void k_locprf(int nprof, int nmu, const double *xmu, int nt, const double *xki,
                         const double *src, const double *rhox, double *ploc, double *work) {
    int p = blockIdx.x * blockDim.x + threadIdx.x;
    if (p >= nprof) return;
    double *d = work + (size_t)p * 3 * nt;
    locprf_one(nmu, xmu, nt, xki + (size_t)p * nt, src + (size_t)p * nt, rhox, d, d + nt, d + 2 * nt,
               ploc + (size_t)p * nmu);
}

void fsg_launch_locprf(cudaStream_t s, int nprof, int nmu, const double *xmu, int nt, const double *xki,
                       const double *src, const double *rhox, double *ploc, double *work) {
    if (nprof > 0) k_locprf<<<(nprof + 127) / 128, 128, 0, s>>>(nprof, nmu, xmu, nt, xki, src, rhox, ploc, work);
}

// ================================================================================================
// MarkWideLines (synth.f90:709-744) over the (packed) line arrays; WlcIdx (synth.f90:677-706)
// ================================================================================================
__device__ __forceinline__ int64_t wlc_idx(const double *wl, double wfirst, int64_t n, double w) {
    if (n == 0 || w < wl[0] - wfirst) return 0;
    int64_t ia = 1, ib = n;
    while (ib - ia > 1) {
        int64_t im = (ia + ib) / 2;
        if (wl[im - 1] - wfirst <= w) ia = im; else ib = im;
    }
    return (wl[ib - 1] - wfirst <= w) ? ib : ia;
}

__global__ void k_mark_wide(AtmView A, int64_t n, const double *wl, int64_t nstep, int32_t *flags,
                            const int32_t *ileft, const int32_t *iright, unsigned long long *nwide) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int f = flags[i];
    if (f & FSG_F_WEAK) return;
    double wr = A.wave[iright[i] - 1], wlft = A.wave[ileft[i] - 1];
    int64_t nrec = wlc_idx(wl, A.wfirst, n, wr) - wlc_idx(wl, A.wfirst, n, wlft) + 1;
    double dv = FSG_VC * (wr - wlft) / ((wl[i] - A.wfirst) + A.wfirst);
    if (nrec > nstep / 2 || dv > 5e3) { flags[i] = f | FSG_F_WIDE; atomicAdd(nwide, 1ull); }
}

void fsg_launch_mark_wide(cudaStream_t s, const AtmView &A, int64_t n, const double *wl, int64_t nstep,
                          int32_t *flags, const int32_t *ileft, const int32_t *iright, unsigned long long *nwide) {
    if (n > 0) k_mark_wide<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(A, n, wl, nstep, flags, ileft, iright, nwide);
}

// ================================================================================================
// Convolution with a short kernel over a spectrum padded with its end values (convol.f90:143-165,
// 206-227, 277-294): out(i) = sum_j in(clamp(i + j - h)) kern(j), h = (n - 1) / 2, in order of j;
// with acc: out(i) = acc(i) + sum * w (the flux sum of the annuli).  One thread per wavelength.
// ================================================================================================
__global__ void k_conv(int nwl, const double *__restrict__ in, int st, const double *__restrict__ kern, int n,
                       double *out, const double *acc, double w) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= nwl) return;
    const int h = (int)((n - 1.0) / 2.0);
    double sm = 0.0;
    for (int j = 0; j < n; j++) {
        int m = min(max(i + j - h, 0), nwl - 1);
        sm = sm + in[(size_t)m * st] * kern[j];
    }
    out[i] = acc ? acc[i] + sm * w : sm;
}

void fsg_launch_conv(cudaStream_t s, int nwl, const double *in, int st, const double *kern, int n, double *out,
                     const double *acc, double w) {
    if (nwl > 0) k_conv<<<(nwl + 255) / 256, 256, 0, s>>>(nwl, in, st, kern, n, out, acc, w);
}


// ================================================================================================
// The reference's elemental line-opacity routines on their own, batched (kernel-level entry points):
// XlineSetup / XlineDepth, LineOpacity1 and LineOpacity2 at given points, AnalyticWindow.  The same
// device functions as the drivers, in the reference's operand order.
// ================================================================================================
// XlineSetup of every line with the drivers' input flags (synth.f90:837-845)
__global__ void k_xline_setup(AtmView A, LineView L, XCoef *xc) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= L.n) return;
    XCoef XC;
    xline_setup(A, L, i, L.wl[i] - A.wfirst, line_input_flags(L, i, 0), &XC);
    xc[i] = XC;
}

// XlineDepth of n lines at every depth: out [n][ntau]
__global__ void k_xline_depth(AtmView A, int64_t n, const XCoef *__restrict__ xc, double *cop, double *vv,
                              double *av) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (g >= n * A.ntau) return;
    const int64_t i = g / A.ntau;
    const int t = (int)(g - i * A.ntau);
    xline_depth(A, t, xc[i], &cop[g], &vv[g], &av[g]);
}

// LineOpacity1 (opacity.f90:297-346) at npts points, one warp per point, lanes over depths
__global__ void k_lineopacity1_pts(AtmView A, BlockView B, int64_t npts, const double *__restrict__ wl,
                                   const int32_t *__restrict__ l1, const int32_t *__restrict__ l2,
                                   const int32_t *__restrict__ iwl, int64_t loff, const float *__restrict__ vtab,
                                   const double *__restrict__ anode, const double *__restrict__ aida, double *out) {
    const int64_t k = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (k >= npts) return;
    const int nt = A.ntau;
    for (int t = lane; t < nt; t += 32) {
        double acc = 0.0;
        for (int64_t il = l1[k]; il <= l2[k]; il++) {
            const int f = B.flags[il - 1];
            if ((f & FSG_F_WEAK) || (f & FSG_F_WIDE) || iwl[k] < B.ileft[il - 1] || iwl[k] > B.iright[il - 1]) continue;
            const int ihe = (f >> 8) & 255;
            const double dWl0 = wl[k] - B.wlcent[il - 1];
            double dWl = dWl0;
            if (ihe > 0) dWl = dWl0 - A.heshf[(ihe - 1) * nt + t];
            const size_t o = (size_t)(il - loff - 1) * nt + t;
            const double V = dWl * B.vv[o];
            const double Vgt = hvoigt64(vtab, anode, aida, B.av[o], V) * B.cop[o];
            acc = acc + Vgt;
        }
        if (A.motype == 1) acc = acc / A.contstd[t];
        out[(size_t)k * nt + t] = acc;
    }
}

// LineOpacity2 (opacity.f90:350-386): point k is line iline[k] at wl[k], grid index iwl[k], with its
// own parameter rows; one thread per (point, depth)
__global__ void k_lineopacity2_pts(AtmView A, BlockView B, int64_t npts, const double *__restrict__ wl,
                                   const int32_t *__restrict__ iline, const int32_t *__restrict__ iwl,
                                   const double *__restrict__ cop, const double *__restrict__ vv,
                                   const double *__restrict__ av, const float *__restrict__ vtab,
                                   const double *__restrict__ anode, const double *__restrict__ aida, double *out) {
    const int64_t g = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    const int nt = A.ntau;
    if (g >= npts * nt) return;
    const int64_t k = g / nt;
    const int t = (int)(g - k * nt);
    const int64_t il = iline[k] - 1;
    const int f = B.flags[il];
    double v = 0.0;
    if (!(f & FSG_F_WEAK) && iwl[k] >= B.ileft[il] && iwl[k] <= B.iright[il]) {
        const int ihe = (f >> 8) & 255;
        const double dWl0 = wl[k] - B.wlcent[il];
        double dWl = dWl0;
        if (ihe > 0) dWl = dWl0 - A.heshf[(ihe - 1) * nt + t];
        const double V = dWl * vv[g];
        v = hvoigt64(vtab, anode, aida, av[g], V) * cop[g];
    }
    if (A.motype == 1) v = v / A.contstd[t];
    out[g] = v;
}

// AnalyticWindow (opacity.f90:678-710) of n lines, one thread per line
__global__ void k_analytic_window(AtmView A, int64_t n, const int32_t *__restrict__ flags,
                                  const double *__restrict__ cop, const double *__restrict__ vv,
                                  const double *__restrict__ av, const double *__restrict__ co, double *dw) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int nt = A.ntau;
    const double iSqrtPi = 0.5641895835477563;
    const int ihe = (flags[i] >> 8) & 255;
    double dWwin = 0.0;
    for (int t = 0; t < nt; t++) {
        const size_t o = (size_t)i * nt + t;
        double r = cop[o] / (A.epsopac * co[o]);
        if (A.motype == 1) r = r / A.contstd[t];
        if (r <= 1.0) continue;
        double w = sqrt(log(r) + fmax(0.0, av[o] * (r * iSqrtPi - av[o]))) / vv[o];
        if (ihe > 0) w = w + fabs(A.heshf[(ihe - 1) * nt + t]);
        dWwin = fmax(dWwin, w);
    }
    dw[i] = dWwin;
}

void fsg_launch_xline_setup(cudaStream_t s, const AtmView &A, const LineView &L, XCoef *xc) {
    if (L.n > 0) k_xline_setup<<<(unsigned)((L.n + 127) / 128), 128, 0, s>>>(A, L, xc);
}
void fsg_launch_xline_depth(cudaStream_t s, const AtmView &A, int64_t n, const XCoef *xc, double *cop, double *vv,
                            double *av) {
    const int64_t m = n * A.ntau;
    if (m > 0) k_xline_depth<<<(unsigned)((m + 127) / 128), 128, 0, s>>>(A, n, xc, cop, vv, av);
}
void fsg_launch_lineopacity1_pts(cudaStream_t s, const AtmView &A, const BlockView &B, int64_t npts, const double *wl,
                                 const int32_t *l1, const int32_t *l2, const int32_t *iwl, int64_t loff,
                                 const VoigtTables &T, double *out) {
    if (npts > 0)
        k_lineopacity1_pts<<<(unsigned)((npts + 7) / 8), 256, 0, s>>>(A, B, npts, wl, l1, l2, iwl, loff, T.vtab,
                                                                      T.anode, T.aida, out);
}
void fsg_launch_lineopacity2_pts(cudaStream_t s, const AtmView &A, const BlockView &B, int64_t npts, const double *wl,
                                 const int32_t *iline, const int32_t *iwl, const double *cop, const double *vv,
                                 const double *av, const VoigtTables &T, double *out) {
    const int64_t m = npts * A.ntau;
    if (m > 0)
        k_lineopacity2_pts<<<(unsigned)((m + 127) / 128), 128, 0, s>>>(A, B, npts, wl, iline, iwl, cop, vv, av,
                                                                       T.vtab, T.anode, T.aida, out);
}
void fsg_launch_analytic_window(cudaStream_t s, const AtmView &A, int64_t n, const int32_t *flags, const double *cop,
                                const double *vv, const double *av, const double *co, double *dw) {
    if (n > 0) k_analytic_window<<<(unsigned)((n + 127) / 128), 128, 0, s>>>(A, n, flags, cop, vv, av, co, dw);
}
