// fsg_magfast.cu -- mixed-precision magnetic line opacity (MagLineOpacity1/3, opacity.f90:391-464,
// 526-591) on wavelength tiles.
//
// MagLineOpac(6, t, lambda) = sum over lines and Zeeman components of (H, L)(a, v_k) LinCop Str_k,
// v_k = (lambda - lambda_c - shift_k) LinVvgt, into the pi / sigma-blue / sigma-red absorption
// (H) and dispersion (L) planes.  A warp owns 32 wavelengths (lanes) x MAG_D depths and takes the tile's
// lines MAG_G at a time: headers, records and components go to its shared memory, then each line's components
// are evaluated in FP32 on depth pairs (packed FMAs) -- outside the line's core range FVoigt's rational
// wing pair, branch-free; inside it the table lerp of FvTab for a < 8, |v| < 8, the wing pair for
// s = v^2 + a^2 >= 196, the two-term continued fraction between (voigt.f90:256-352) -- summed per line in
// FP32 and added to FP64 accumulators.  The per-(line, depth) records come from the FP64 XlineDepth values
// (k_mag_params_fast).
//
// The wing pair is H = a/sqrt(pi) (u + a^2 + 1/2) / D, L = v/sqrt(pi) (u + a^2 - 1/2) / D with u = v^2 and
// D = s^2 - v^2 + a^2 + 1/4 = u (u + 2a^2 - 1) + (a^2 + 1/2)^2 (voigt.f90:280-289): eleven FP32 operations
// (half as many issued, packed) and one reciprocal per component and point.  5,000 Zeeman lines on 50,001
// wavelengths (4.3e10 component evaluations), 56 depths: 34 ms, against 50 ms for CTAs of eight warps of
// four depths that read each line's header, records and components from global memory and evaluated in
// scalar FP32.  Issue slots (61 %), the FP32 pipe (43 %) and the reciprocal pipe (37 %; a third of it the
// conversions of the sums) are all well loaded and none is full.  Tried beside it: four depths per warp (158
// registers, 35 ms), one copy of the component loops for the three profiles (42 ms), components staged once per
// CTA behind barriers (38 ms).
#include "fsg_fp64.cuh"
#include "fsg_tile.cuh"

#define MAG_D 2                       // depths per warp
#define MAG_G 8                       // lines per group
#define MAG_W 4                       // warps per CTA
#define MAG_C 32                      // components staged per line; longer lists are read in place

// Wing records of two neighbouring depths side by side, as the scalar wing pass has them (wing_pairs(ntau)
// per line; the last half of an odd count is 0): LinVvgt, a, LinCop
struct __align__(8) MagPair { float vv[2], a[2], cop[2]; };
// table / continued-fraction region: a, LinCop, the table row ia (1-based, 0: a >= 8) and its weight ua
struct __align__(16) MagCore { float a, cop, ua; int ia; };
// Zeeman components of a block line in ZView
struct __align__(16) MagComp { int64_t pi, si; int np, ns; int pad[2]; };

// Records of a block's lines, and per line its header with the core range [cl, cr]: every wavelength
// of the window where some depth and Zeeman component may have s = v^2 + a^2 < 196 (half-width
// max_t sqrt(196.05 - a^2) / LinVvgt, + the largest |component shift| and |He I shift|, + one
// wavelength); outside it every point takes FVoigt's rational wing pair.  One warp per line, lanes over depths.
__global__ void __launch_bounds__(128)
k_mag_params_fast(AtmView A, LineView L, ZView Z, const int64_t *__restrict__ idx, int64_t j0,
                  int64_t nb, const int32_t *__restrict__ flags, const int32_t *__restrict__ ileft,
                  const int32_t *__restrict__ iright, const double *__restrict__ anode,
                  const double *__restrict__ aida, MagPair *pairs, MagCore *core, LineHdr *hdr, MagComp *comp) {
    const int64_t j = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int lane = threadIdx.x & 31;
    if (j >= nb) return;                                // whole warps leave together
    const int64_t i = idx[j0 + j];
    const int nt = A.ntau, np = wing_pairs(nt);
    const int f = flags[i];
    const double wlc = L.wl[i] - A.wfirst;
    XCoef XC;
    xline_setup(A, L, i, wlc, f, &XC);
    const float an1 = (float)anode[1], ai0 = (float)aida[0];
    const int ihe = (f >> 8) & 255;
    double hcore = -1.0, shmax = 0.0;
    for (int t = lane; t < 2 * np; t += 32) {
        MagPair &m = pairs[(size_t)j * np + (t >> 1)];
        const int e = t & 1;
        if (t >= nt) { m.vv[e] = m.a[e] = m.cop[e] = 0.0f; continue; }
        double cop, vv, av;
        xline_depth(A, t, XC, &cop, &vv, &av);
        const double q = 196.05 - av * av;
        if (q > 0.0) hcore = fmax(hcore, sqrt(q) / vv * (1.0 + 1e-5));
        if (ihe > 0) shmax = fmax(shmax, fabs(A.heshf[(size_t)(ihe - 1) * nt + t]));
        if (A.motype == 1) cop = cop / A.contstd[t];
        m.vv[e] = (float)vv; m.a[e] = (float)av; m.cop[e] = (float)cop;
        MagCore r;
        r.cop = (float)cop; r.a = (float)av;
        if (!(r.a < 8.0f)) { r.ia = 0; r.ua = 0.0f; }
        else if (r.a < an1) { r.ia = 1; r.ua = r.a * ai0; }
        else {
            int ia = min((int)(sqrtf(r.a) * 141.42135623730951f) + 1, FSG_NVA);
            r.ia = ia;
            r.ua = (r.a - (float)anode[ia - 1]) * (float)aida[ia - 1];
        }
        core[(size_t)j * nt + t] = r;
    }
    double zmax = 0.0;
    for (int k = lane; k < Z.npi[i]; k += 32) zmax = fmax(zmax, fabs((double)Z.splpi[Z.pi_off[i] + k]));
    for (int k = lane; k < Z.nsi[i]; k += 32) zmax = fmax(zmax, fabs((double)Z.splsi[Z.si_off[i] + k]));
    for (int o = 16; o > 0; o >>= 1) {
        hcore = fmax(hcore, __shfl_xor_sync(0xffffffffu, hcore, o));
        shmax = fmax(shmax, __shfl_xor_sync(0xffffffffu, shmax, o));
        zmax = fmax(zmax, __shfl_xor_sync(0xffffffffu, zmax, o));
    }
    if (lane != 0) return;
    LineHdr h;
    h.wlh = (float)wlc;
    h.wll = (float)(wlc - (double)h.wlh);
    h.ileft = ileft[i]; h.iright = iright[i];
    h.cl = 1; h.cr = 0;
    if (hcore >= 0.0) {
        const double half = hcore + zmax + shmax;
        int a = lower_index(A.wave, A.nwl, wlc - half) + 1;
        int b = lower_index(A.wave, A.nwl, wlc + half);
        if (b < A.nwl && A.wave[b] == wlc + half) b++;
        const int cl = max(a - 1, h.ileft), cr = min(b + 1, h.iright);
        if (cl <= cr) { h.cl = cl; h.cr = cr; }
    }
    h.silent = ihe;                                   // He I table index (0: none)
    h.pairable = 0;
    hdr[j] = h;
    comp[j] = MagComp{ Z.pi_off[i], Z.si_off[i], Z.npi[i], Z.nsi[i], { 0, 0 } };
}

__device__ __forceinline__ float rcp_approx_m(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// FVoigt (H, L) in FP32 at v (signed), L odd in v.  The table lerp takes each row's two v nodes in one
// 16-byte load (fvtab2); the wing and continued-fraction forms take one approximate reciprocal.
__device__ __forceinline__ void fv32(const float4 *__restrict__ fvtab2, const MagCore &r, float v, float &H, float &L) {
    const float av = fabsf(v), a = r.a, a2 = a * a, v2 = av * av, s = v2 + a2;
    if (r.ia > 0 && av < 8.0f) {
        const float fv = av * 125.0f;
        const int iv = min((int)fv, FSG_NVV - 1);
        const float tv = fv - (float)iv;
        const float4 *p0 = fvtab2 + (r.ia - 1) * FSG_NV1 + iv;
        const float4 g0 = __ldg(p0), g1 = __ldg(p0 + FSG_NV1);      // (H_i, L_i, H_i+1, L_i+1) of rows ia, ia+1
        const float h0 = g0.x + tv * (g0.z - g0.x), h1 = g1.x + tv * (g1.z - g1.x);
        const float l0 = g0.y + tv * (g0.w - g0.y), l1 = g1.y + tv * (g1.w - g1.y);
        H = h0 + r.ua * (h1 - h0);
        L = l0 + r.ua * (l1 - l0);
    } else if (s >= 196.0f) {
        const float w = 0.56418958354775628f * rcp_approx_m(s * s - v2 + a2 + 0.25f);
        H = w * a * (s + 0.5f);
        L = w * av * (s - 0.5f);
    } else {
        const float p = v2 - a2 - 1.5f, q = 2.0f * av * a;
        const float dr = av * p - a * q, di = av * q + a * p;
        const float w = 0.56418958354775628f * rcp_approx_m(dr * dr + di * di);
        H = w * ((p + 0.5f) * di - q * dr);
        L = w * ((p + 0.5f) * dr + q * di);
    }
    L = copysignf(fabsf(L), v);
}

// component k of a line: pi components, then sigma
__device__ __forceinline__ float2 mag_component(const ZView &Z, const MagComp &c, int k) {
    const bool pi = k < c.np;
    const float sp = pi ? Z.splpi[c.pi + k] : Z.splsi[c.si + k - c.np];
    const float st = pi ? Z.strpi[c.pi + k] : Z.strsi[c.si + k - c.np];
    return make_float2(-sp, st);
}

// the line's components through f(component, profile): pi into profile 0, the blue half of sigma into 1, the
// red into 2; the staged ones from shared memory, the rest of a longer list in place
#define MAG_COMPONENTS(f) do { \
        const float2 *zc = z_s[warp][q]; \
        int k = 0; \
        _Pragma("unroll 2") for (; k < min(k1, MAG_C); k++) f(zc[k], 0); \
        for (; k < k1; k++) f(mag_component(Z, c, k), 0); \
        _Pragma("unroll 2") for (; k < min(k2, MAG_C); k++) f(zc[k], 1); \
        for (; k < k2; k++) f(mag_component(Z, c, k), 1); \
        _Pragma("unroll 2") for (; k < min(k3, MAG_C); k++) f(zc[k], 2); \
        for (; k < k3; k++) f(mag_component(Z, c, k), 2); \
    } while (0)

struct MagJob {
    int ntau, nwl, ntiles;
    const double *wave;
    const LineHdr *hdr;
    const MagPair *pairs;
    const MagCore *core;
    const MagComp *comp;
    const double *heshf;
    const int *tile_lo, *tile_hi;
    const float4 *fvtab2;
    double *mlo;
};

__global__ void __launch_bounds__(32 * MAG_W) k_mag_fast(MagJob J, ZView Z) {
    constexpr int NP = MAG_D / 2;
    __shared__ int queue_s[MAG_W][64];
    __shared__ LineHdr hdr_s[MAG_W][MAG_G];
    __shared__ MagComp comp_s[MAG_W][MAG_G];
    __shared__ MagPair pair_s[MAG_W][MAG_G][NP];
    __shared__ float2 z_s[MAG_W][MAG_G][MAG_C];          // (-shift, strength): pi components, then sigma
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int ntau = J.ntau, ng = (ntau + MAG_D - 1) / MAG_D, npair = wing_pairs(ntau);
    const int64_t item = (int64_t)blockIdx.x * MAG_W + warp;
    if (item >= (int64_t)J.ntiles * ng) return;          // warps are independent: no CTA barrier below
    const int tile = (int)(item / ng), t0 = (int)(item % ng) * MAG_D;
    const int lo = J.tile_lo[tile], hi = J.tile_hi[tile];
    if (lo > hi) return;
    const int nd = min(MAG_D, ntau - t0);
    const int p = tile * 32 + lane, p1 = p + 1;
    const int tile_first = tile * 32 + 1, tile_last = min(tile * 32 + 32, J.nwl);
    const double wd = J.wave[min(p, J.nwl - 1)];
    const float wvh = (float)wd, wvl = (float)(wd - (double)wvh);
    const int *queue = queue_s[warp];
    double acc[MAG_D][6];
#pragma unroll
    for (int d = 0; d < MAG_D; d++)
#pragma unroll
        for (int q = 0; q < 6; q++) acc[d][q] = 0.0;
    auto group = [&](int head, int n) {
        if (lane < n) {
            const int row = queue[(head + lane) & 63];
            hdr_s[warp][lane] = J.hdr[row];
            comp_s[warp][lane] = J.comp[row];
        }
        for (int e = lane; e < n * NP; e += 32) {
            const int q = e / NP, pr = (t0 >> 1) + e % NP;
            MagPair v = {};
            if (pr < npair) v = J.pairs[(size_t)queue[(head + q) & 63] * npair + pr];
            pair_s[warp][q][e % NP] = v;
        }
        __syncwarp();
        for (int q = 0; q < n; q++) {
            const MagComp c = comp_s[warp][q];
            if (lane < c.np + c.ns && lane < MAG_C) z_s[warp][q][lane] = mag_component(Z, c, lane);
        }
        __syncwarp();
        for (int q = 0; q < n; q++) {
            const LineHdr h = hdr_s[warp][q];
            const MagComp c = comp_s[warp][q];
            const float dl = (wvh - h.wlh) + (wvl - h.wll);
            const bool in = p1 >= h.ileft && p1 <= h.iright;
            float2 vv[NP], vb[NP], s[NP][6];
#pragma unroll
            for (int j = 0; j < NP; j++) {
                const MagPair &m = pair_s[warp][q][j];
                vv[j] = make_float2(m.vv[0], m.vv[1]);
                float2 d2 = make_float2(dl, dl);
                if (h.silent > 0) {
                    const double *sh = J.heshf + (size_t)(h.silent - 1) * ntau;
                    d2.x -= (float)sh[min(t0 + 2 * j, ntau - 1)];
                    d2.y -= (float)sh[min(t0 + 2 * j + 1, ntau - 1)];
                }
                vb[j] = __fmul2_rn(d2, vv[j]);
#pragma unroll
                for (int r = 0; r < 6; r++) s[j][r] = make_float2(0.0f, 0.0f);
            }
            const int k1 = c.np, k2 = c.np + c.ns / 2, k3 = c.np + c.ns;
            if (h.cl > h.cr || h.cr < tile_first || h.cl > tile_last) {
                float2 b1[NP], b0[NP], ah[NP], am[NP];
#pragma unroll
                for (int j = 0; j < NP; j++) {
                    const MagPair &m = pair_s[warp][q][j];
                    const float2 a2 = make_float2(m.a[0] * m.a[0], m.a[1] * m.a[1]);
                    b1[j] = make_float2(2.0f * a2.x - 1.0f, 2.0f * a2.y - 1.0f);
                    ah[j] = make_float2(a2.x + 0.5f, a2.y + 0.5f);
                    am[j] = make_float2(a2.x - 0.5f, a2.y - 0.5f);
                    b0[j] = __fmul2_rn(ah[j], ah[j]);
                }
                auto one = [&](const float2 z, int r) {
                    const float2 ns = make_float2(z.x, z.x), st = make_float2(z.y, z.y);
#pragma unroll
                    for (int j = 0; j < NP; j++) {
                        const float2 v = __ffma2_rn(ns, vv[j], vb[j]);
                        const float2 u = __fmul2_rn(v, v);
                        const float2 den = __ffma2_rn(u, __fadd2_rn(u, b1[j]), b0[j]);
                        const float2 rr = make_float2(rcp_approx_m(den.x), rcp_approx_m(den.y));
                        s[j][r] = __ffma2_rn(st, __fmul2_rn(__fadd2_rn(u, ah[j]), rr), s[j][r]);
                        s[j][r + 3] = __ffma2_rn(st, __fmul2_rn(__fmul2_rn(__fadd2_rn(u, am[j]), rr), v), s[j][r + 3]);
                    }
                };
                MAG_COMPONENTS(one);
                if (in) {
#pragma unroll
                    for (int j = 0; j < NP; j++) {
                        const MagPair &m = pair_s[warp][q][j];
                        const float2 ch = make_float2(0.56418958354775628f * m.a[0] * m.cop[0], 0.56418958354775628f * m.a[1] * m.cop[1]);
                        const float2 cv = make_float2(0.56418958354775628f * m.cop[0], 0.56418958354775628f * m.cop[1]);
#pragma unroll
                        for (int r = 0; r < 3; r++) {
                            const float2 a = __fmul2_rn(s[j][r], ch), b = __fmul2_rn(s[j][r + 3], cv);
                            acc[2 * j][r] += (double)a.x; acc[2 * j + 1][r] += (double)a.y;
                            acc[2 * j][r + 3] += (double)b.x; acc[2 * j + 1][r + 3] += (double)b.y;
                        }
                    }
                }
            } else if (in) {
                const int row = queue[(head + q) & 63];
                MagCore m[MAG_D];
#pragma unroll
                for (int d = 0; d < MAG_D; d++) m[d] = J.core[(size_t)row * ntau + t0 + min(d, nd - 1)];
                auto one = [&](const float2 z, int r) {
#pragma unroll
                    for (int d = 0; d < MAG_D; d++) {
                        const float vvd = d & 1 ? vv[d >> 1].y : vv[d >> 1].x, vbd = d & 1 ? vb[d >> 1].y : vb[d >> 1].x;
                        float H, L;
                        fv32(J.fvtab2, m[d], fmaf(z.x, vvd, vbd), H, L);
                        float2 &sa = s[d >> 1][r], &sb = s[d >> 1][r + 3];
                        if (d & 1) { sa.y = fmaf(z.y, H, sa.y); sb.y = fmaf(z.y, L, sb.y); }
                        else { sa.x = fmaf(z.y, H, sa.x); sb.x = fmaf(z.y, L, sb.x); }
                    }
                };
                MAG_COMPONENTS(one);
#pragma unroll
                for (int d = 0; d < MAG_D; d++)
#pragma unroll
                    for (int r = 0; r < 6; r++) {
                        const float x = d & 1 ? s[d >> 1][r].y : s[d >> 1][r].x;
                        acc[d][r] += (double)(x * m[d].cop);
                    }
            }
        }
        __syncwarp();                                    // the group's shared records may be replaced
    };
    tile_lines<MAG_G>(J.hdr, lo, hi, tile_first, tile_last, queue_s[warp], lane, group);
    if (p >= J.nwl) return;
#pragma unroll
    for (int d = 0; d < MAG_D; d++) {
        if (d >= nd) break;
        double *dst = J.mlo + ((size_t)p * ntau + t0 + d) * 6;
#pragma unroll
        for (int q = 0; q < 6; q++) dst[q] = dst[q] + acc[d][q];
    }
}

// a block's records for nb lines of nt depths, the parts of widest alignment first: components | cores | pairs
static MagCore *mag_cores(void *rec, int64_t nb) { return (MagCore *)((MagComp *)rec + nb); }
static MagPair *mag_pairs(void *rec, int64_t nb, int nt) { return (MagPair *)(mag_cores(rec, nb) + (size_t)nb * nt); }
static_assert(sizeof(MagComp) % alignof(MagCore) == 0 && sizeof(MagCore) % alignof(MagPair) == 0, "aligned parts");

// bytes of a line's records
size_t fsg_mag_rec_bytes(int nt) { return sizeof(MagPair) * wing_pairs(nt) + sizeof(MagCore) * nt + sizeof(MagComp); }

void fsg_launch_mag_params_fast(cudaStream_t s, const AtmView &A, const LineView &L, const ZView &Z, const int64_t *idx,
                                int64_t j0, int64_t nb, const int32_t *flags, const int32_t *il, const int32_t *ir,
                                const VoigtTables &T, void *rec, LineHdr *hdr) {
    if (nb > 0)
        k_mag_params_fast<<<(unsigned)((nb + 3) / 4), 128, 0, s>>>(A, L, Z, idx, j0, nb, flags, il, ir, T.anode, T.aida,
                                                                  mag_pairs(rec, nb, A.ntau), mag_cores(rec, nb), hdr,
                                                                  (MagComp *)rec);
}

int fsg_launch_mag_fast(cudaStream_t s, const AtmView &A, const LineHdr *hdr, void *rec, int64_t nb, const ZView &Z,
                        const int *tlo, const int *thi, const VoigtTables &T, double *mlo) {
    const int ntiles = (A.nwl + 31) / 32;
    MagJob J{ A.ntau, A.nwl, ntiles, A.wave, hdr, mag_pairs(rec, nb, A.ntau), mag_cores(rec, nb), (const MagComp *)rec,
              A.heshf, tlo, thi, T.fvtab2, mlo };
    const int64_t items = (int64_t)ntiles * ((A.ntau + MAG_D - 1) / MAG_D);
    k_mag_fast<<<(unsigned)((items + MAG_W - 1) / MAG_W), 32 * MAG_W, 0, s>>>(J, Z);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}
