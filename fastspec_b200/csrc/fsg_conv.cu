// fsg_conv.cu -- disk integration with broadening (convol.f90:67-300) in one pass over the spectrum.
//
// Per annulus: rotation, then radial-tangential macroturbulence, each a short kernel over the spectrum padded
// with its end values, then the flux sum; at the end the Gaussian of the flux.  A CTA owns CONV_T wavelengths
// of one kind (line, continuum): for every annulus it stages the intensities with the halo both kernels need,
// convolves from shared memory to shared memory and adds to the flux kept in registers.  A thread forms
// CONV_R consecutive points, so a staged value serves CONV_R taps' products; the odd stride between lanes
// keeps the loads free of bank conflicts.
//
// Bound by launches and latency as a kernel per annulus, kernel and kind (44 launches, strided loads of the
// intensities, 305 us for 200,001 wavelengths, 7 annuli, 25 / 4 km/s and R = 65,000); two launches here.
#include "fsg_internal.cuh"

#define CONV_R 5
#define CONV_TH 128
#define CONV_T (CONV_R * CONV_TH)

// out[o] = sum_j in[o + j] taps[j], j < n, for the CONV_R outputs from o on
__device__ __forceinline__ void taps_sum(const double *in, const double *__restrict__ taps, int n, double (&acc)[CONV_R]) {
    double v[CONV_R];
#pragma unroll
    for (int r = 0; r < CONV_R; r++) { acc[r] = 0.0; v[r] = in[r]; }
#pragma unroll 5
    for (int j = 0; j < n; j++) {
        const double k = __ldg(taps + j);
#pragma unroll
        for (int r = 0; r < CONV_R; r++) acc[r] = fma(v[r], k, acc[r]);
#pragma unroll
        for (int r = 0; r + 1 < CONV_R; r++) v[r] = v[r + 1];
        v[CONV_R - 1] = in[j + CONV_R];
    }
}

// Annulus im: rotation taps taps[roff .. roff + rn) (rn = 0: none) and macroturbulence taps[moff .. + mn);
// odd counts.  Intensities [nwl][stride] per kind.
struct ConvJob {
    int nwl, stride, nann, rh, mh;         // rh, mh: the largest half-widths of either kind of kernel
    int roff[16], rn[16], moff[16], mn[16];
    double w[16];
    const double *in[2];
    double *out[2];
    const double *taps;
};

// shared memory: staged intensities [CONV_T + 2 (rh + mh) + pad] | rotated ones [CONV_T + 2 mh + pad]
static size_t conv_smem(int rh, int mh) {
    return sizeof(double) * (size_t)(2 * CONV_T + 2 * rh + 4 * mh + 8 * CONV_R);
}

__global__ void __launch_bounds__(CONV_TH) k_disk_conv(ConvJob J) {
    extern __shared__ double sm[];
    const int p0 = blockIdx.x * CONV_T, kind = blockIdx.y, nwl = J.nwl;
    const double *__restrict__ in = J.in[kind];
    double *a = sm, *b = sm + CONV_T + 2 * (J.rh + J.mh) + 2 * CONV_R;
    double flux[CONV_R];
#pragma unroll
    for (int r = 0; r < CONV_R; r++) flux[r] = 0.0;
    const int o0 = threadIdx.x * CONV_R;
    for (int im = 0; im < J.nann; im++) {
        const int rn = J.rn[im], mn = J.mn[im], rh = rn / 2, mh = mn / 2;
        const int na = CONV_T + 2 * (rh + mh), nb = CONV_T + 2 * mh;
        for (int e = threadIdx.x; e < na + 2 * CONV_R; e += CONV_TH) {
            const int p = min(max(p0 - mh - rh + e, 0), nwl - 1);
            a[e] = in[(size_t)p * J.stride + im];
        }
        __syncthreads();
        const double *s = a;
        if (rn) {
            // the rotated spectrum at p0 - mh + o; where that lies outside the grid the nearest end's value
            for (int o = o0; o < nb; o += CONV_T) {
                double acc[CONV_R];
                taps_sum(a + o, J.taps + J.roff[im], rn, acc);
#pragma unroll
                for (int r = 0; r < CONV_R; r++) if (o + r < nb) b[o + r] = acc[r];
            }
            __syncthreads();
            const int lo = max(mh - p0, 0), hi = min(nwl - 1 - p0 + mh, nb - 1);   // the grid's ends in b
            for (int e = threadIdx.x; e < nb + 2 * CONV_R; e += CONV_TH)
                if (e < lo || e > hi) b[e] = b[e < lo ? lo : hi];
            __syncthreads();
            s = b;
        }
        double acc[CONV_R];
        if (mn) taps_sum(s + o0, J.taps + J.moff[im], mn, acc);
        else
#pragma unroll
            for (int r = 0; r < CONV_R; r++) acc[r] = s[o0 + r];
#pragma unroll
        for (int r = 0; r < CONV_R; r++) flux[r] = fma(acc[r], J.w[im], flux[r]);
        __syncthreads();                                 // a and b are free for the next annulus
    }
#pragma unroll
    for (int r = 0; r < CONV_R; r++)
        if (p0 + o0 + r < nwl) J.out[kind][p0 + o0 + r] = flux[r];
}

// The broadened flux of both kinds: intensities spl/spc [nwl][nmu], taps on the device, annulus im's kernels
// as in ConvJob; the Gaussian taps[goff .. goff + gn) (gn = 0: none) last, through the work arrays tl, tc [nwl].
// CONV_WIDE (positive; errors are negative): kernels too wide, nothing was launched, the caller convolves annulus by
// annulus.
//
// Where that is: a CTA rotates the halo of the macroturbulence too, rn (CONV_T + 2 mh) products for rn CONV_T, and wide
// kernels leave room for few CTAs on an SM and little L1 for the taps.  Time annulus by annulus over fused, 200,001
// wavelengths, 3 and 9 annuli, by the half-widths (rotation, macroturbulence); the fused pass's products over the
// others; CTAs per SM:
//   (100, 600) 3.3, 3.8 x; 1.3; 7    (1200, 600) 1.6, 1.8 x; 2.3; 4    (600, 2000) 1.2, 1.3 x; 2.4; 2
//   (1200, 2000) 0.96, 1.1 x; 3.3; 2    (2500, 2000) 0.48, 0.58 x; 4.5; 2    (6000, 200) 1.1, 1.3 x; 1.6; 2
//   (0, 6000) 1.3, 1.6 x; 1.0; 1    (100, 5000) 1.1, 1.1 x; 1.3; 1    (300, 5000) 0.96, 1.0 x; 1.9; 1
int fsg_launch_disk_conv(cudaStream_t s, int nwl, int nmu, const double *spl, const double *spc, const double *taps,
                         const int *roff, const int *rn, const int *moff, const int *mn, const double *wmu, int goff,
                         int gn, double *tl, double *tc, double *sfl, double *sfc) {
    ConvJob J;
    if (nmu > (int)(sizeof J.rn / sizeof *J.rn)) return CONV_WIDE;
    J.nwl = nwl; J.stride = nmu; J.nann = nmu; J.rh = J.mh = 0; J.taps = taps;
    for (int im = 0; im < nmu; im++) {
        J.roff[im] = roff[im]; J.rn[im] = rn[im]; J.moff[im] = moff[im]; J.mn[im] = mn[im]; J.w[im] = wmu[im];
        J.rh = rn[im] / 2 > J.rh ? rn[im] / 2 : J.rh;
        J.mh = mn[im] / 2 > J.mh ? mn[im] / 2 : J.mh;
    }
    const size_t sm1 = conv_smem(J.rh, J.mh), sm2 = conv_smem(0, gn / 2), most = 200 * 1024;
    if (sm1 > most || sm2 > most) return CONV_WIDE;
    double fused = 0.0, apart = 0.0;                     // products of a CTA's wavelengths
    for (int im = 0; im < nmu; im++) {
        fused += (double)rn[im] * (CONV_T + mn[im]) + (double)mn[im] * CONV_T;
        apart += ((double)rn[im] + mn[im]) * CONV_T;
    }
    const int ctas = (int)((227 * 1024) / (sm1 + 1024)), taps_most = 2 * (J.rh > J.mh ? J.rh : J.mh);
    if (fused > (ctas < 2 ? 1.4 : ctas == 2 && taps_most > 4096 ? 1.65 : 2.5) * apart) return CONV_WIDE;
    const size_t sm = sm1 > sm2 ? sm1 : sm2;
    if (sm > 48 * 1024 &&
        cudaFuncSetAttribute(k_disk_conv, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)most) != cudaSuccess)
        return FSG_E_CUDA;
    const dim3 grid((nwl + CONV_T - 1) / CONV_T, 2);
    J.in[0] = spl; J.in[1] = spc;
    J.out[0] = gn ? tl : sfl; J.out[1] = gn ? tc : sfc;
    k_disk_conv<<<grid, CONV_TH, sm1, s>>>(J);
    if (gn) {                                            // ConvolGau of the flux (convol.f90:236-240)
        J.stride = 1; J.nann = 1; J.rh = 0; J.mh = gn / 2;
        J.rn[0] = 0; J.moff[0] = goff; J.mn[0] = gn; J.w[0] = 1.0;
        J.in[0] = tl; J.in[1] = tc; J.out[0] = sfl; J.out[1] = sfc;
        k_disk_conv<<<grid, CONV_TH, sm2, s>>>(J);
    }
    return cudaPeekAtLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}
