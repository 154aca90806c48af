// fsg_accum64.cu -- plain FP64 line opacity on wavelength tiles: LineOpacity1 (opacity.f90:297-346) with the
// wide lines (synth.f90:981-1001), and MagLineOpacity1/3 (opacity.f90:391-464, 526-591).
//
//   LineOpac(t, p) += sum over lines l with Ileft(l) <= p <= Iright(l) of HVoigt(a(l,t), v) LinCop(l,t)
//
// A warp owns 32 P wavelengths (lanes) x D depths and takes the lines of its tile in list order, so
// every point sums its lines in the reference's order whatever the tile or the wavelength range of the
// call.  Warps share nothing: each reads the windows of the tile's candidate lines 32 at a time, queues
// those that touch the tile and works through the queue 32 / D lines at a time.  For a group the lanes
// first turn the lines' (LinCop, LinVvgt, LinAvgt) at the warp's depths into the wing form's
// coefficients, one (line, depth) per lane, in shared memory; then every lane evaluates its points:
//   outside the line's core range (s >= 196 at every depth, voigt.f90:100-101)
//     val = c1 (t + 1) / (t^2 + 2 a^2),  t = dl^2 LinVvgt^2 + a^2 - 1/2,  c1 = LinCop a / sqrt(pi)
//     -- three FMAs, a reciprocal of three more, one FMA into the sum;
//   inside it the same form where t >= 195.5, else the table lerp or the continued fraction of HVoigt.
// He I lines with a Stark shift per depth take the point-by-point form over their whole window.
//
// Bound by the FP64 pipe: 7.5 FP64 instructions per wing evaluation (64 lanes/clk/SM: 2.5e12
// evaluations/s).  P = 2 and D = 4 keep the per-line work (offsets, window test, 8 shared loads) under a
// tenth of the evaluations' and leave registers for six 4-warp CTAs per SM.  20,000 lines, 40,001 wavelengths, 56
// depths (4.7e9 evaluations): 4.0 ms, against 15.9 ms for a warp per wavelength with lanes over depths and 13.3 ms
// more for the wide lines of a pass of their own.  Half of the FP64 cycles are used.  Six CTAs per SM (78 registers);
// five take 2 % longer, four 7 %, and the next group's loads in flight gained nothing.
#include "fsg_fp64.cuh"
#include "fsg_tile.cuh"

#define A64_W 4                     // warps per CTA

struct Wing64 { double vv2, c2m1, twoA, c1; };
struct Core64 { double vv, a, ua, cop; int ia, pad; };

// The wing term's numerator n and reciprocal r.  It is added as fma(n, r, sum) in every branch that takes it, so that a
// point's sum does not depend on how its tile or range cuts the line's window.
struct Wing64Term { double n, r; };
__device__ __forceinline__ Wing64Term wing64(double t, const Wing64 &w) {
    return { fma(w.c1, t, w.c1), rcp64(fma(t, t, w.twoA)) };
}

// HVoigt (voigt.f90:81-107) where s < 196, table row and weight of a given
__device__ __forceinline__ double core64(const float *__restrict__ vtab, const Core64 &c, double av) {
    if (c.ia > 0 && av < 8.0) {
        const double fv = av * 125.0;
        const int iv = min((int)fv, FSG_NVV - 1);
        const double tv = fv - (double)iv;
        const float *p0 = vtab + (c.ia - 1) * FSG_NV1 + iv, *p1 = p0 + FSG_NV1;
        const float t00 = __ldg(p0), t01 = __ldg(p0 + 1), t10 = __ldg(p1), t11 = __ldg(p1 + 1);
        const double c0 = (double)t00 + tv * (double)(t01 - t00), c1 = (double)t10 + tv * (double)(t11 - t10);
        return c0 + c.ua * (c1 - c0);
    }
    const double a2 = c.a * c.a, v2 = av * av, p = v2 - a2 - 1.5, q = 2.0 * av * c.a;
    const double dr = av * p - c.a * q, di = av * q + c.a * p;
    return FSG_SQRTPIINV * ((p + 0.5) * di - q * dr) / (dr * dr + di * di);
}

// table row and weight of a as HVoigt takes them (voigt.f90:84-92); ia = 0: a >= 8
__device__ __forceinline__ void table_row64(const double *__restrict__ anode, const double *__restrict__ aida, double a,
                                            int &ia, double &ua) {
    if (!(a < 8.0)) { ia = 0; ua = 0.0; }
    else if (a < anode[1]) { ia = 1; ua = __dmul_rn(a, aida[0]); }
    else {
        ia = min((int)(sqrt(a) * (1.0 / (2.8284271247461903 / 400.0))) + 1, FSG_NVA);
        ua = __dmul_rn(a - anode[ia - 1], aida[ia - 1]);
    }
}

struct Accum64Job {
    int ntau, nwl, w0, w1;              // wavelengths w0 .. w1 (1-based) are filled
    int tile0, ntiles, ngrp;            // first tile, tiles, depth groups
    const double *wave;
    const LineHdr64 *hdr;
    const double3 *p64;
    const int *lo, *hi;                 // candidate rows of each 32 wavelengths of the grid
    const double *heshf, *contstd, *anode, *aida;
    const float *vtab;
    double *lineopac;
};

// P wavelengths per lane, D depths per warp, 32 / D lines per group: one (line, depth) pair per lane
template <int P, int D>
__global__ void __launch_bounds__(32 * A64_W, 6) k_accum64(Accum64Job J) {
    constexpr int G = 32 / D, TW = 32 * P;
    __shared__ int queue_s[A64_W][64];
    __shared__ __align__(16) LineHdr64 hdr_s[A64_W][G];
    __shared__ __align__(16) Wing64 wing_s[A64_W][G][D];
    __shared__ Core64 core_s[A64_W][G][D];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t item = (int64_t)blockIdx.x * A64_W + warp;
    if (item >= (int64_t)J.ntiles * J.ngrp) return;      // warps are independent: no CTA barrier below
    const int tile = J.tile0 + (int)(item / J.ngrp), t0 = (int)(item % J.ngrp) * D;
    const int ntau = J.ntau, lo = J.lo[tile * P], hi = J.hi[min(tile * P + P, (J.nwl + 31) / 32) - 1];
    if (lo > hi) return;
    const int first = max(tile * TW + 1, J.w0), last = min(tile * TW + TW, J.w1);
    const int *queue = queue_s[warp];
    double wv[P], acc[P][D];
    int pix[P];                                      // 1-based
#pragma unroll
    for (int k = 0; k < P; k++) {
        pix[k] = tile * TW + lane + 32 * k + 1;
        wv[k] = J.wave[min(pix[k], J.nwl) - 1];
#pragma unroll
        for (int d = 0; d < D; d++) acc[k][d] = 0.0;
    }
    const int tq = lane / D, td = lane % D;      // this lane's (line, depth) of a group
    auto group = [&](int head, int n) {                  // n <= G queued lines from head on
        const bool mine = tq < n;
        const int row = mine ? queue[(head + tq) & 63] : 0;
        LineHdr64 h;
        if (mine) {
            h = J.hdr[row];
            if (td == 0) hdr_s[warp][tq] = h;
            Wing64 w = { 0.0, 1.0e3, 0.0, 0.0 };         // past the last depth: a term of 0
            if (t0 + td < ntau) {
                const double3 p = J.p64[(size_t)row * ntau + t0 + td];
                const double a2 = __dmul_rn(p.z, p.z);
                w.vv2 = p.y * p.y; w.c2m1 = a2 - 0.5; w.twoA = 2.0 * a2; w.c1 = p.x * p.z * FSG_SQRTPIINV;
                if (h.ihe > 0 || (h.cl <= h.cr && h.cr >= first && h.cl <= last)) {
                    Core64 c;
                    c.vv = p.y; c.a = p.z; c.cop = p.x; c.pad = 0;
                    table_row64(J.anode, J.aida, p.z, c.ia, c.ua);
                    core_s[warp][tq][td] = c;
                }
            }
            wing_s[warp][tq][td] = w;
        }
        __syncwarp();
        for (int q = 0; q < n; q++) {
            const LineHdr64 g = hdr_s[warp][q];
            double dl[P], x[P];
#pragma unroll
            for (int k = 0; k < P; k++) { dl[k] = wv[k] - g.wlc; x[k] = __dmul_rn(dl[k], dl[k]); }
            if (g.ihe > 0 || (g.cl <= g.cr && g.cr >= first && g.cl <= last)) {
                const int nd = min(D, ntau - t0);
#pragma unroll
                for (int d = 0; d < D; d++) {
                    if (d >= nd) break;
                    const Wing64 w = wing_s[warp][q][d];
                    const double sh = g.ihe > 0 ? J.heshf[(size_t)(g.ihe - 1) * ntau + t0 + d] : 0.0;
#pragma unroll
                    for (int k = 0; k < P; k++) {
                        if (pix[k] < g.il || pix[k] > g.ir) continue;
                        const double dk = dl[k] - sh, t = fma(__dmul_rn(dk, dk), w.vv2, w.c2m1);
                        const Core64 &c = core_s[warp][q][d];
                        if (t >= 195.5) {
                            const Wing64Term v = wing64(t, w);
                            acc[k][d] = fma(v.n, v.r, acc[k][d]);
                        } else acc[k][d] = fma(core64(J.vtab, c, fabs(dk) * c.vv), c.cop, acc[k][d]);
                    }
                }
            } else if (g.il <= first && g.ir >= last) {
#pragma unroll
                for (int d = 0; d < D; d++) {
                    const Wing64 w = wing_s[warp][q][d];
#pragma unroll
                    for (int k = 0; k < P; k++) {
                        const Wing64Term v = wing64(fma(x[k], w.vv2, w.c2m1), w);
                        acc[k][d] = fma(v.n, v.r, acc[k][d]);
                    }
                }
            } else {
                bool in[P];
#pragma unroll
                for (int k = 0; k < P; k++) in[k] = pix[k] >= g.il && pix[k] <= g.ir;
#pragma unroll
                for (int d = 0; d < D; d++) {
                    const Wing64 w = wing_s[warp][q][d];
#pragma unroll
                    for (int k = 0; k < P; k++) {
                        const Wing64Term v = wing64(fma(x[k], w.vv2, w.c2m1), w);
                        if (in[k]) acc[k][d] = fma(v.n, v.r, acc[k][d]);
                    }
                }
            }
        }
        __syncwarp();                                    // the group's shared records may be replaced
    };
    tile_lines<G>(J.hdr, lo, hi, first, last, queue_s[warp], lane, group);
#pragma unroll
    for (int k = 0; k < P; k++) {
        if (pix[k] < J.w0 || pix[k] > J.w1) continue;
        double *dst = J.lineopac + (size_t)(pix[k] - 1) * ntau + t0;
#pragma unroll
        for (int d = 0; d < D; d++)
            if (t0 + d < ntau) dst[d] += J.contstd ? acc[k][d] / J.contstd[t0 + d] : acc[k][d];
    }
}

static Accum64Job accum64_job(const AtmView &A, const LineHdr64 *hdr, const double3 *p64, const int *lo, const int *hi,
                              int w0, int w1, int tw, int depths, const VoigtTables &T, double *out) {
    Accum64Job J;
    J.ntau = A.ntau; J.nwl = A.nwl; J.w0 = w0; J.w1 = w1;
    J.tile0 = (w0 - 1) / tw;
    J.ntiles = (w1 - 1) / tw - J.tile0 + 1;
    J.ngrp = (A.ntau + depths - 1) / depths;
    J.wave = A.wave; J.hdr = hdr; J.p64 = p64; J.lo = lo; J.hi = hi;
    J.heshf = A.heshf; J.contstd = A.motype == 1 ? A.contstd : nullptr;
    J.anode = T.anode; J.aida = T.aida; J.vtab = T.vtab; J.lineopac = out;
    return J;
}

// Few wavelengths: with 64 x 4 points a warp few warps set out, and the pass is the latency of one warp's lines (20,000 lines
// on 301 wavelengths, 56 depths: 70 warps, 23.6 ms; a warp per wavelength with lanes over depths 18.3 ms).  32 x 1
// points a warp make eight times as many (4.7 ms), 32 x 2 four times (7.5 ms).  A point's sum is the same in every
// form, bit for bit.  6,000 lines, 56 depths, ms of the forms 32 x 1, 32 x 2, 64 x 4: 3,001 wavelengths (658 warps of the
// last) 0.95, 0.98, 1.77; 6,001 (1,316) 1.30, 1.20, 1.36; 8,001 (1,764) 1.51, 1.23, 1.22.
#define A64_FEW11 660
#define A64_FEW12 1600

template <int P, int D>
static int launch_accum64(cudaStream_t s, const AtmView &A, const LineHdr64 *hdr, const double3 *p64, const int *lo,
                          const int *hi, int w0, int w1, const VoigtTables &T, double *lineopac) {
    const Accum64Job J = accum64_job(A, hdr, p64, lo, hi, w0, w1, 32 * P, D, T, lineopac);
    const int64_t items = (int64_t)J.ntiles * J.ngrp;
    k_accum64<P, D><<<(unsigned)((items + A64_W - 1) / A64_W), 32 * A64_W, 0, s>>>(J);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

// rows hdr / p64 with the row ranges lo / hi of each 32 wavelengths of the whole grid onto LineOpac at the
// wavelengths w0 .. w1 (1-based, inclusive)
int fsg_launch_accum64(cudaStream_t s, const AtmView &A, const LineHdr64 *hdr, const double3 *p64, const int *lo,
                       const int *hi, int w0, int w1, const VoigtTables &T, double *lineopac) {
    if (w1 < w0) return FSG_OK;
    const int64_t warps = (int64_t)((w1 - w0) / 64 + 1) * ((A.ntau + 3) / 4);
    if (warps < A64_FEW11) return launch_accum64<1, 1>(s, A, hdr, p64, lo, hi, w0, w1, T, lineopac);
    if (warps < A64_FEW12) return launch_accum64<1, 2>(s, A, hdr, p64, lo, hi, w0, w1, T, lineopac);
    return launch_accum64<2, 4>(s, A, hdr, p64, lo, hi, w0, w1, T, lineopac);
}

// ---- magnetic lines ----------------------------------------------------------------------------------
// MagLineOpac(6, t, p) += sum over lines and Zeeman components of (H, L)(a, v_k) LinCop Str_k with
// v_k = (lambda - lambda_c - shift_k) LinVvgt, into the pi, blue and red absorption (H) and dispersion (L)
// profiles.  As k_accum64 with one wavelength per lane and one or two depths per warp (six sums each).  Outside
// the line's core range (Zeeman shifts included) a component takes FVoigt's rational pair (voigt.f90:280-289)
//   u = v^2, D = u (u + 2 a^2 - 1) + (a^2 + 1/2)^2,  H = a/sqrt(pi) h,  L = v/sqrt(pi) (h - 1/D),
//   h = (u + a^2 + 1/2) / D
// in 13 FP64 instructions (the FP64 pipe bounds it); LinCop a/sqrt(pi) and LinCop/sqrt(pi) multiply the
// line's six sums once.  700 lines, 6,001 wavelengths, 56 depths: 2.5 ms, against 8.1 ms for a warp per wavelength and
// pass; a quarter of it is the core form.
struct MagWing64 { double vv, b1, b0, ah, ch, cv; };

// FVoigt's (H, L) where s < 196 (voigt.f90:256-352), L odd in v
__device__ __forceinline__ void fcore64(const float2 *__restrict__ ftab, const Core64 &c, double v, double &H, double &L) {
    const double av = fabs(v);
    if (c.ia > 0 && av < 8.0) {
        const double fv = av * 125.0;
        const int iv = min((int)fv, FSG_NVV - 1);
        const double tv = fma(av, 125.0, -(double)iv);
        const float2 *p0 = ftab + (c.ia - 1) * FSG_NV1 + iv, *p1 = p0 + FSG_NV1;
        const float2 t00 = __ldg(p0), t01 = __ldg(p0 + 1), t10 = __ldg(p1), t11 = __ldg(p1 + 1);
        const double h0 = fma(tv, (double)(t01.x - t00.x), (double)t00.x), h1 = fma(tv, (double)(t11.x - t10.x), (double)t10.x);
        const double l0 = fma(tv, (double)(t01.y - t00.y), (double)t00.y), l1 = fma(tv, (double)(t11.y - t10.y), (double)t10.y);
        H = fma(c.ua, h1 - h0, h0);
        L = fma(c.ua, l1 - l0, l0);
    } else {
        const double p = fma(av, av, -__dmul_rn(c.a, c.a)) - 1.5, q = __dmul_rn(2.0 * av, c.a);
        const double dr = fma(av, p, -__dmul_rn(c.a, q)), di = fma(av, q, __dmul_rn(c.a, p));
        const double w = FSG_SQRTPIINV / fma(dr, dr, __dmul_rn(di, di));
        H = w * fma(p + 0.5, di, -__dmul_rn(q, dr));
        L = w * fma(p + 0.5, dr, __dmul_rn(q, di));
    }
    L = copysign(fabs(L), v);
}

template <int D>
__global__ void __launch_bounds__(32 * A64_W, 5) k_mag64(Accum64Job J, ZView Z, const float2 *__restrict__ ftab) {
    constexpr int G = 32 / D;
    __shared__ int queue_s[A64_W][64];
    __shared__ __align__(16) LineHdr64 hdr_s[A64_W][G];
    __shared__ MagWing64 wing_s[A64_W][G][D];
    __shared__ Core64 core_s[A64_W][G][D];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int64_t item = (int64_t)blockIdx.x * A64_W + warp;
    if (item >= (int64_t)J.ntiles * J.ngrp) return;      // warps are independent: no CTA barrier below
    const int tile = J.tile0 + (int)(item / J.ngrp), t0 = (int)(item % J.ngrp) * D;
    const int ntau = J.ntau, lo = J.lo[tile], hi = J.hi[tile];
    if (lo > hi) return;
    const int first = max(tile * 32 + 1, J.w0), last = min(tile * 32 + 32, J.w1);
    const int *queue = queue_s[warp];
    const int pix = tile * 32 + lane + 1;                // 1-based
    const double wv = J.wave[min(pix, J.nwl) - 1];
    double acc[D][6];
#pragma unroll
    for (int d = 0; d < D; d++)
#pragma unroll
        for (int r = 0; r < 6; r++) acc[d][r] = 0.0;
    const int tq = lane / D, td = lane % D;      // this lane's (line, depth) of a group
    auto group = [&](int head, int n) {
        if (tq < n) {
            const int row = queue[(head + tq) & 63];
            const LineHdr64 h = J.hdr[row];
            if (td == 0) hdr_s[warp][tq] = h;
            MagWing64 w = { 0.0, 0.0, 1.0, 0.0, 0.0, 0.0 };
            if (t0 + td < ntau) {
                const double3 p = J.p64[(size_t)row * ntau + t0 + td];
                const double a2 = __dmul_rn(p.z, p.z);
                w.vv = p.y; w.b1 = 2.0 * a2 - 1.0; w.ah = a2 + 0.5; w.b0 = w.ah * w.ah;
                w.cv = p.x * FSG_SQRTPIINV; w.ch = w.cv * p.z;
                Core64 c;
                c.vv = p.y; c.a = p.z; c.cop = p.x; c.pad = 0;
                if (h.cl <= h.cr && h.cr >= first && h.cl <= last) table_row64(J.anode, J.aida, p.z, c.ia, c.ua);
                core_s[warp][tq][td] = c;
            }
            wing_s[warp][tq][td] = w;
        }
        __syncwarp();
        for (int q = 0; q < n; q++) {
            const LineHdr64 g = hdr_s[warp][q];
            const double dl = wv - g.wlc;
            const bool in = pix >= g.il && pix <= g.ir;
            const int np = Z.npi[g.zi], ns = Z.nsi[g.zi], nsh = ns / 2;
            const float *spi = Z.splpi + Z.pi_off[g.zi], *ssi = Z.splsi + Z.si_off[g.zi];
            const float *rpi = Z.strpi + Z.pi_off[g.zi], *rsi = Z.strsi + Z.si_off[g.zi];
            double vv[D], vb[D], s[D][6];
#pragma unroll
            for (int d = 0; d < D; d++) {
                const int t = min(t0 + d, ntau - 1);
                const double sh = g.ihe > 0 ? J.heshf[(size_t)(g.ihe - 1) * ntau + t] : 0.0;
                vv[d] = wing_s[warp][q][d].vv;
                vb[d] = __dmul_rn(dl - sh, vv[d]);
#pragma unroll
                for (int r = 0; r < 6; r++) s[d][r] = 0.0;
            }
            if (g.cl > g.cr || g.cr < first || g.cl > last) {
                double b1[D], b0[D], ah[D];
#pragma unroll
                for (int d = 0; d < D; d++) {
                    b1[d] = wing_s[warp][q][d].b1; b0[d] = wing_s[warp][q][d].b0; ah[d] = wing_s[warp][q][d].ah;
                }
                auto comps = [&](const float *sp_, const float *st_, int k0, int k1, int r) {
                    for (int k = k0; k < k1; k++) {
                        const double sp = (double)sp_[k], st = (double)st_[k];
#pragma unroll
                        for (int d = 0; d < D; d++) {
                            const double v = fma(-sp, vv[d], vb[d]), u = __dmul_rn(v, v), ua = u + ah[d];
                            const double rr = rcp64(fma(u, u + b1[d], b0[d]));
                            s[d][r] = fma(st, __dmul_rn(ua, rr), s[d][r]);
                            s[d][r + 3] = fma(st, __dmul_rn(fma(ua, rr, -rr), v), s[d][r + 3]);
                        }
                    }
                };
                comps(spi, rpi, 0, np, 0);
                comps(ssi, rsi, 0, nsh, 1);
                comps(ssi, rsi, nsh, ns, 2);
                if (in) {
#pragma unroll
                    for (int d = 0; d < D; d++) {
                        const double ch = wing_s[warp][q][d].ch, cv = wing_s[warp][q][d].cv;
#pragma unroll
                        for (int r = 0; r < 3; r++) {
                            acc[d][r] = fma(s[d][r], ch, acc[d][r]);
                            acc[d][r + 3] = fma(s[d][r + 3], cv, acc[d][r + 3]);
                        }
                    }
                }
            } else if (in) {
                auto comps = [&](const float *sp_, const float *st_, int k0, int k1, int r) {
                    for (int k = k0; k < k1; k++) {
                        const double sp = (double)sp_[k], st = (double)st_[k];
#pragma unroll
                        for (int d = 0; d < D; d++) {
                            if (t0 + d >= ntau) break;
                            const Core64 &c = core_s[warp][q][d];
                            const double v = fma(-sp, vv[d], vb[d]), u = __dmul_rn(v, v);
                            double H, L;
                            if (fma(c.a, c.a, u) >= 196.0) {
                                const MagWing64 &w = wing_s[warp][q][d];
                                const double rr = rcp64(fma(u, u + w.b1, w.b0)), ua = u + w.ah;
                                H = FSG_SQRTPIINV * c.a * __dmul_rn(ua, rr); L = FSG_SQRTPIINV * fma(ua, rr, -rr) * v;
                            } else fcore64(ftab, c, v, H, L);
                            s[d][r] = fma(st, H, s[d][r]);
                            s[d][r + 3] = fma(st, L, s[d][r + 3]);
                        }
                    }
                };
                comps(spi, rpi, 0, np, 0);
                comps(ssi, rsi, 0, nsh, 1);
                comps(ssi, rsi, nsh, ns, 2);
#pragma unroll
                for (int d = 0; d < D; d++) {
                    if (t0 + d >= ntau) break;
                    const double cop = core_s[warp][q][d].cop;
#pragma unroll
                    for (int r = 0; r < 6; r++) acc[d][r] = fma(s[d][r], cop, acc[d][r]);
                }
            }
        }
        __syncwarp();                                    // the group's shared records may be replaced
    };
    tile_lines<G>(J.hdr, lo, hi, first, last, queue_s[warp], lane, group);
    if (pix < J.w0 || pix > J.w1) return;
#pragma unroll
    for (int d = 0; d < D; d++) {
        if (t0 + d >= ntau) break;
        double *dst = J.lineopac + ((size_t)(pix - 1) * ntau + t0 + d) * 6;
#pragma unroll
        for (int r = 0; r < 6; r++) dst[r] += J.contstd ? acc[d][r] / J.contstd[t0 + d] : acc[d][r];
    }
}

// One depth a warp where the warps of two would not fill the GPU one and a half times (2,960 are resident): 200 lines, 56
// depths, 301 wavelengths 1.58 -> 0.90 ms, 4,001 0.72 -> 0.65; 3,000 lines, 40,001 wavelengths 32.4 ms with two, 38.4 with
// one.  A point's sum is the same in either form, bit for bit.
#define M64_FEW 4440

template <int D>
static int launch_mag64(cudaStream_t s, const AtmView &A, const LineHdr64 *hdr, const double3 *p64, const ZView &Z,
                        const int *lo, const int *hi, int w0, int w1, const VoigtTables &T, double *mlo) {
    const Accum64Job J = accum64_job(A, hdr, p64, lo, hi, w0, w1, 32, D, T, mlo);
    const int64_t items = (int64_t)J.ntiles * J.ngrp;
    k_mag64<D><<<(unsigned)((items + A64_W - 1) / A64_W), 32 * A64_W, 0, s>>>(J, Z, T.fvtab);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

// as fsg_launch_accum64, onto MagLineOpac
int fsg_launch_mag64(cudaStream_t s, const AtmView &A, const LineHdr64 *hdr, const double3 *p64, const ZView &Z,
                     const int *lo, const int *hi, int w0, int w1, const VoigtTables &T, double *mlo) {
    if (w1 < w0) return FSG_OK;
    const int64_t warps = (int64_t)((w1 - w0) / 32 + 1) * ((A.ntau + 1) / 2);
    if (warps < M64_FEW) return launch_mag64<1>(s, A, hdr, p64, Z, lo, hi, w0, w1, T, mlo);
    return launch_mag64<2>(s, A, hdr, p64, Z, lo, hi, w0, w1, T, mlo);
}
