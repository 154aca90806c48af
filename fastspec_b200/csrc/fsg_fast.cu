// fsg_fast.cu -- mixed-precision line-opacity accumulation (FP32 Voigt, compensated sums).
//
// The work of LineopCalc's accumulation (LineOpacity1, opacity.f90:297-346) is
//   LineOpac(t, p) = sum over retained lines l with Ileft(l) <= p <= Iright(l) of
//                    HVoigt(a(l,t), (lambda_p - lambda_l) / dlD(l,t)) * LinCop(l,t).
// It is split by the branch HVoigt takes.  Each line has a core range (every wavelength of its
// window where some depth may have s = v^2 + a^2 < 196); outside it every depth takes the
// reference's rational wing form (voigt.f90:100-101).
//
// Wing pass (k_accum_fast): a warp owns a tile of TW = 32 P wavelengths x D depths, lane l the
// wavelengths tile0 + l + 32k (k < P).  It picks the tile's lines from the candidate range and brings their
// headers and records to shared memory a group at a time, the next group's loads in flight while it works
// through the present one; each thread keeps P x D FP32 partials over FOLD lines, folded into Kahan (sum,
// compensation) pairs in shared memory.  Lines are binned by window width (class c holds windows of up to
// 256 * 2^c wavelengths), a tile range for each class, so a tile's candidate range stays close to the lines
// that touch it; narrow classes use 64-wavelength tiles, wide ones 128.
//
// Core pass (k_core_fast): over the core ranges, 32-wavelength tiles x 8 depths per warp, the points where s < 196: the
// table lerp (|v| < 8, a < 8) or the two-term continued fraction (voigt.f90:103-107), exactly as
// HVoigt branches.  No atomics; one read-modify-write of the FP64 LineOpac per tile and launch;
// deterministic order.
#include "fsg_internal.cuh"
#include "fsg_mbar.cuh"

#include <cub/device/device_scan.cuh>
#include <cuda/functional>
#include <algorithm>

#define CLASS_W0 128      // class c: windows of at most CLASS_W0 * 2^(c+1) wavelengths

// HVoigt in FP32 outside the table (a >= 8 or |v| >= 8, s < 196): the two-term continued
// fraction of voigt.f90:103-107 at |v| = av
__device__ __forceinline__ float hv_cf32(float av, float a) {
    float a2 = a * a, v2 = av * av;
    float p = v2 - a2 - 1.5f, q = 2.0f * av * a;
    float dr = av * p - a * q, di = av * q + a * p;
    float r;                                            // the denominator is of the order of v^6: no subnormals
    asm("div.approx.ftz.f32 %0, %1, %2;" : "=f"(r) : "f"((p + 0.5f) * di - q * dr), "f"(dr * dr + di * di));
    return 0.56418958354775628f * r;
}

// Kahan-compensated accumulation of one value
#define KAHAN(S, CC, V) do { float _y = (V) - (CC); float _t = (S) + _y; (CC) = (_t - (S)) - _y; (S) = _t; } while (0)

// Lines folded into the compensated sums at a time: each thread adds up to FOLD lines into FP32
// register partials, then Kahan-adds every partial into its (sum, compensation) pair in shared
// memory.  The partials carry at most FOLD terms, so their rounding stays at the FP32 unit
// roundoff of a few terms; the Kahan pairs carry the long sums.
#define FOLD 32
// cp.async.bulk moves multiples of 16 bytes between 16-byte aligned addresses
static_assert(sizeof(LineHdr) % 16 == 0 && sizeof(CoreRec) % 16 == 0, "bulk-copied records: multiples of 16 bytes");

__device__ __forceinline__ float rcp_approx(float x) {
    float r;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(r) : "f"(x));
    return r;
}

// Wing pass.  Every window point where fl32(t) >= 195.5 (s >= 196) takes HVoigt's rational wing
// form:
//   val = c1 (t + 1) / (t^2 + twoA),  t = dl^2 vv2 + c2m1
// (three FMAs, one reciprocal, one FMA into the partial sum).  Outside the line's core range [cl, cr]
// that is every depth.  Lines whose window covers the whole tile outside their core range (the common
// case for wide windows) need no mask, and two of them share a reciprocal:
//   n0 / d0 + n1 / d1 = (n0 d1 + n1 d0) / (d0 d1).
// For the others the points outside the window get an x for which the term is exactly 0.  On tiles that meet
// the core range, each point whose t is below 195.5 (table or continued fraction, the core pass's share) has
// its t replaced by 1e19, whose term is exactly 0 too: the two passes split the points by the same FP32 test,
// so each point is evaluated once.
//
// What bounds it: the reciprocal unit takes 8 cycles a warp and evaluation, the four FMAs 4; paired, 4 and 5 (a
// loop of nothing else reaches 8.5 and 6.9).  Eight depths x 4 wavelengths a lane halve the record loads per
// evaluation against 4 x 4, sixteen lines a group the staging against 8: a million lines, 483,000 wavelengths, 56 depths
// 44.9 -> 40.3 ms (single, 4 x 4) -> 33.0 ms (pairs, 8 x 4, 16 lines).
//
// A pair rounds in other places than two single terms, three products more and one addition less; against 64 bits it is
// no further off (rms of LineOpac 4.8e-8 with pairs, 5.0e-8 without, for 20,000 lines over 200 A; 3.8 and 4.0e-8 for 1e6
// molecular lines).  The two roundings differ most where few lines make up a pixel: by 5e-9 of the flux at 140 lines per
// pixel, 1.3e-9 at 240, 4e-10 at 500, 4e-11 at 2,100.  The pass is short there, and tiles that fewer than WING_PAIR_MIN
// lines touch take them one at a time.  Lines are counted, not candidates, so that a tile sums alike whatever
// part of the list and of the grid a call has; the count ends at WING_PAIR_MIN.

// A line as the warp's group holds it: {wlh, wll, code, xm}.  code: first and last wavelength of the window
// inside the tile (bits 0-7, 8-15), WING_CORE (a core range meets it); xm: the x that silences a point.
#define WING_CORE (1 << 16)
#define WING_G 16                     // lines per group
#define WING_PAIR_MIN 1024

// shared memory of one warp
template <int D, int P>
struct __align__(16) WingWarp {
    float4 rec[WING_G][D];            // D / 2 depth pairs of two float4
    float4 hdr[WING_G];
    float2 ksum[D * P][32];           // Kahan (sum, compensation)
    int queue[64];
};

// One tile and depth group (depths t0 .. t0 + D - 1, t0 a multiple of D) of one job, by one warp; warps
// share nothing.  The arithmetic is packed FP32 on depth pairs.
template <int D, int P>
__device__ __forceinline__ void wing_tile(const WingJob &J, int tile, int t0, WingWarp<D, P> &S, int lane) {
    constexpr int TW = 32 * P, NP = D / 2, U = WING_G * D / 32;      // U: record loads per lane and group
    const int ntau = J.ntau, nwl = J.nwl, units = 2 * wing_pairs(ntau);
    int64_t ncand = 0;                                  // lines that may touch the tile
    for (int sg = 0; sg < J.nseg; sg++)
        ncand += max(J.tile_hi[sg * J.seg_stride + tile] - J.tile_lo[sg * J.seg_stride + tile] + 1, 0);
    if (!ncand) return;
    const float4 *__restrict__ wing = (const float4 *)J.wing;
    const int p0 = tile * TW;
    // wavelength offsets as FP32 hi + lo: dl = (wvh - wlh) + (wvl - wll) keeps dl to FP32 relative
    // accuracy next to the line centre
    float wvh[P], wvl[P];
#pragma unroll
    for (int k = 0; k < P; k++) {
        double w = J.wave[min(p0 + lane + 32 * k, nwl - 1)];
        wvh[k] = (float)w;
        wvl[k] = (float)(w - (double)wvh[k]);
    }
    float2 part[NP][P];
#pragma unroll
    for (int j = 0; j < NP; j++)
#pragma unroll
        for (int k = 0; k < P; k++) {
            part[j][k] = make_float2(0.0f, 0.0f);
            S.ksum[2 * (j * P + k)][lane] = make_float2(0.0f, 0.0f);
            S.ksum[2 * (j * P + k) + 1][lane] = make_float2(0.0f, 0.0f);
        }
    int nfold = 0;
    const int tile_first = p0 + 1, tile_last = min(p0 + TW, nwl);
    int touch = 0;                                      // lines that touch the tile, counted up to WING_PAIR_MIN
    for (int sg = 0; ncand >= WING_PAIR_MIN && touch < WING_PAIR_MIN && sg < J.nseg; sg++) {
        const int last = J.tile_hi[sg * J.seg_stride + tile];
        for (int b = J.tile_lo[sg * J.seg_stride + tile]; b <= last && touch < WING_PAIR_MIN; b += 128)
#pragma unroll
            for (int u = 0; u < 4; u++) {
                const int i = b + 32 * u + lane;
                const int2 w = i <= last ? *(const int2 *)&J.hdr[i].ileft : make_int2(1, 0);
                touch += __popc(__ballot_sync(0xffffffffu, w.y >= tile_first && w.x <= tile_last));
            }
    }
    const bool pairs = touch >= WING_PAIR_MIN;
    float4 rnext[U], hnext;                             // the next group's records and (lanes < n) header
    int nnext = 0, npair = 0, slot = 0;                            // lines; lane q's line's place in the group
    auto fetch = [&](int head, int n) {
        nnext = n;
        bool pair = false;
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = lane + 32 * u, q = e / D, i = t0 + e % D;
            rnext[u] = make_float4(0.0f, 0.0f, 0.0f, 0.0f);          // past the last depth: never stored
            if (q < n && i < units) rnext[u] = __ldg(wing + (size_t)S.queue[(head + q) & 63] * units + i);
        }
        if (lane < n) {
            const LineHdr h = J.hdr[S.queue[(head + lane) & 63]];
            const bool core_hit = h.cl <= h.cr && h.cr >= tile_first && h.cl <= tile_last;
            const bool full = h.ileft <= tile_first && h.iright >= tile_last && !core_hit;
            const int l = max(h.ileft - tile_first, 0), r = min(h.iright - tile_first, TW - 1);
            hnext = make_float4(h.wlh, h.wll, __int_as_float(l | r << 8 | (core_hit ? WING_CORE : 0)),
                                __int_as_float(h.silent));
            pair = pairs && full && h.pairable;
        }
        // the lines to be paired first
        const unsigned pm = __ballot_sync(0xffffffffu, pair), before = __popc(pm & ((1u << lane) - 1u));
        npair = __popc(pm);
        slot = pair ? before : npair + lane - before;
    };
    auto stage = [&](int m) {                              // the fetched group into shared memory
        __syncwarp();                                   // every lane is done with the group before
#pragma unroll
        for (int u = 0; u < U; u++) {
            const int e = lane + 32 * u;
            S.rec[__shfl_sync(0xffffffffu, slot, e / D)][e % D] = rnext[u];
        }
        if (lane < m) S.hdr[slot] = hnext;
        __syncwarp();
    };
    auto fold = [&]() {                                 // the partials into the Kahan pairs
        nfold = 0;
#pragma unroll
        for (int j = 0; j < NP; j++)
#pragma unroll
            for (int k = 0; k < P; k++) {
                float2 s0 = S.ksum[2 * (j * P + k)][lane], s1 = S.ksum[2 * (j * P + k) + 1][lane];
                KAHAN(s0.x, s0.y, part[j][k].x);
                KAHAN(s1.x, s1.y, part[j][k].y);
                S.ksum[2 * (j * P + k)][lane] = s0;
                S.ksum[2 * (j * P + k) + 1][lane] = s1;
                part[j][k] = make_float2(0.0f, 0.0f);
            }
    };
    auto flush = [&]() {                                // the Kahan pairs onto LineOpac
#pragma unroll
        for (int k = 0; k < P; k++) {
            const int pix = p0 + lane + 32 * k;
            double *dst = J.lineopac + (size_t)pix * ntau + t0;
#pragma unroll
            for (int d = 0; d < D; d++) {
                float2 &ks = S.ksum[2 * ((d >> 1) * P + k) + (d & 1)][lane];
                if (pix < nwl && t0 + d < ntau) dst[d] += (double)ks.x - (double)ks.y;
                ks = make_float2(0.0f, 0.0f);
            }
        }
    };
    auto offsets = [&](float4 h, float (&x)[P]) {       // x = dl^2 of the lane's wavelengths
#pragma unroll
        for (int k = 0; k < P; k++) {
            const float dl = (wvh[k] - h.x) + (wvl[k] - h.y);
            x[k] = dl * dl;
        }
    };
    auto work = [&](int n, int np) {
        int q = 0;
        for (; q + 1 < np; q += 2) {                    // full lines, two at a time
            float x0[P], x1[P];
            offsets(S.hdr[q], x0);
            offsets(S.hdr[q + 1], x1);
#pragma unroll
            for (int j = 0; j < NP; j++) {
                const float4 a0 = S.rec[q][2 * j], b0 = S.rec[q][2 * j + 1];
                const float4 a1 = S.rec[q + 1][2 * j], b1 = S.rec[q + 1][2 * j + 1];
                const float2 c0 = make_float2(b0.z, b0.w), c1 = make_float2(b1.z, b1.w);
#pragma unroll
                for (int k = 0; k < P; k++) {
                    const float2 t0 = __ffma2_rn(make_float2(x0[k], x0[k]), make_float2(a0.x, a0.y), make_float2(a0.z, a0.w));
                    const float2 t1 = __ffma2_rn(make_float2(x1[k], x1[k]), make_float2(a1.x, a1.y), make_float2(a1.z, a1.w));
                    const float2 d0 = __ffma2_rn(t0, t0, make_float2(b0.x, b0.y)), d1 = __ffma2_rn(t1, t1, make_float2(b1.x, b1.y));
                    const float2 n0 = __ffma2_rn(c0, t0, c0), n1 = __ffma2_rn(c1, t1, c1);
                    const float2 den = __fmul2_rn(d0, d1), num = __ffma2_rn(n0, d1, __fmul2_rn(n1, d0));
                    part[j][k] = __ffma2_rn(num, make_float2(rcp_approx(den.x), rcp_approx(den.y)), part[j][k]);
                }
            }
        }
        for (; q < n; q++) {
            const float4 h = S.hdr[q];
            const int code = __float_as_int(h.z);
            float x[P];
            offsets(h, x);
            // points outside the window take the header's offset x, for which the wing term is exactly 0
            const int l = code & 255, r = code >> 8 & 255;
#pragma unroll
            for (int k = 0; k < P; k++) {
                const int p = lane + 32 * k;
                x[k] = (p >= l && p <= r) ? x[k] : h.w;
            }
            const bool core_hit = code & WING_CORE;
#pragma unroll
            for (int j = 0; j < NP; j++) {
                const float4 a = S.rec[q][2 * j], b = S.rec[q][2 * j + 1];
                const float2 vv2 = make_float2(a.x, a.y), c2m1 = make_float2(a.z, a.w);
                const float2 twoA = make_float2(b.x, b.y), c1 = make_float2(b.z, b.w);
#pragma unroll
                for (int k = 0; k < P; k++) {
                    float2 t = __ffma2_rn(make_float2(x[k], x[k]), vv2, c2m1);
                    if (core_hit) {                     // the core pass's points
                        t.x = t.x < 195.5f ? 1.0e19f : t.x;
                        t.y = t.y < 195.5f ? 1.0e19f : t.y;
                    }
                    const float2 den = __ffma2_rn(t, t, twoA), num = __ffma2_rn(c1, t, c1);
                    part[j][k] = __ffma2_rn(num, make_float2(rcp_approx(den.x), rcp_approx(den.y)), part[j][k]);
                }
            }
        }
        nfold += n;
        if (nfold > FOLD - WING_G) fold();
    };
    // One loop, so that each of the forms above stands in the code once: lines into the queue, a group of them
    // into flight, the group before through the arithmetic.
    int head = 0, cnt = 0, sg = 0, base = 0, hi = -1;
    bool open = false, some = false;                    // lines of segment sg are left to look at; some are not on LineOpac
    for (;;) {
        while (cnt < WING_G) {
            if (!open) {
                if (sg == J.nseg || (J.fold_seg && (cnt || nnext || some))) break;
                base = J.tile_lo[sg * J.seg_stride + tile];
                hi = J.tile_hi[sg * J.seg_stride + tile];
                sg++;
                open = base <= hi;
                continue;
            }
            const int i = base + lane;
            bool sel = false;
            if (i <= hi) {
                const int2 w = *(const int2 *)&J.hdr[i].ileft;
                sel = w.y >= tile_first && w.x <= tile_last;
            }
            base += 32;
            open = base <= hi;
            const unsigned m = __ballot_sync(0xffffffffu, sel);
            if (sel) S.queue[(head + cnt + __popc(m & ((1u << lane) - 1u))) & 63] = i;
            cnt += __popc(m);
        }
        __syncwarp();
        const int n = min(cnt, WING_G);
        const int m = nnext, mp = npair;
        nnext = 0;
        if (m) stage(m);
        if (n) fetch(head, n);
        head += n;
        cnt -= n;
        if (m) work(m, mp);
        some = some || m;
        if (!n && !m) {                               // nothing in flight: the tile's lines, or this segment's, end here
            const bool last = sg == J.nseg && !open;
            if (nfold) fold();
            if (some) flush();
            some = false;
            if (last) break;
        }
    }
}

#define WING_D 8                      // depths per warp
#define WING_W 4                      // warps per CTA
#define FEW_MAX 592
#define WING_BW 8                     // warps per CTA of the persistent form

// one (tile, depth group) per warp, the groups of a tile in turn
template <int D, int P>
__global__ void __launch_bounds__(32 * WING_W, P == 2 ? 5 : 4)
k_accum_fast(WingJob J, int ntiles) {
    __shared__ WingWarp<D, P> S[WING_W];
    const int warp = threadIdx.x >> 5, ng = (J.ntau + D - 1) / D;
    const int64_t item = (int64_t)blockIdx.x * WING_W + warp;
    if (item >= (int64_t)ntiles * ng) return;           // warps are independent: no CTA barrier
    wing_tile<D, P>(J, (int)(item / ng), (int)(item % ng) * D, S[warp], threadIdx.x & 31);
}

// Persistent form for many jobs (batched atmospheres): warps take (job, tile, depth group) items from a
// device work queue (*queue, zero at launch) until all are done; item0[j] is the first item of job j
// (prefix sums of the jobs' tiles x groups, item0[njobs] = total).
template <int D, int P>
__global__ void __launch_bounds__(32 * WING_BW, 2)
k_accum_batch(const WingJob *__restrict__ jobs, const int *__restrict__ item0, int njobs, unsigned *queue) {
    extern __shared__ __align__(128) unsigned char smem_raw[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    WingWarp<D, P> &S = ((WingWarp<D, P> *)smem_raw)[warp];
    const int total = item0[njobs];
    for (;;) {
        int item = 0;
        if (lane == 0) item = (int)atomicAdd(queue, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= total) break;
        int a = 0, b = njobs - 1;                          // job with item0[a] <= item < item0[a + 1]
        while (a < b) { int m = (a + b + 1) >> 1; if (item0[m] <= item) a = m; else b = m - 1; }
        const WingJob J = jobs[a];
        const int ng = (J.ntau + D - 1) / D, r = item - item0[a];
        wing_tile<D, P>(J, r / ng, (r % ng) * D, S, lane);
    }
}

// Tile width per window-width class: narrow windows get narrower tiles so fewer lanes idle.
int fsg_class_pix(int cls) { return cls <= 1 ? 2 : 4; }

// depth groups of the wing pass
int fsg_wing_groups(int ntau) { return (ntau + WING_D - 1) / WING_D; }

// Few tiles: at eight depths a warp their warps would not fill a quarter of the 148 x 16 that are resident, so the pass
// is the latency of its longest warp.  Two depths a warp then make four times as many of them, which set out together.
// A depth's sum is the same in either form.  300 lines, 1,001 wavelengths: core pass 51 -> 25 us, wing pass 54 -> 31 us.
static bool few_tiles(int ntiles, int ntau) { return (int64_t)ntiles * ((ntau + 7) / 8) < FEW_MAX; }

// the wing pass of one job on tiles of 32 P wavelengths
int fsg_launch_accum_fast(cudaStream_t st, int P, const WingJob &J) {
    const int TW = 32 * P, ntiles = (J.nwl + TW - 1) / TW;
    const bool few = few_tiles(ntiles, J.ntau);
    const int D = few ? 2 : WING_D;
    const unsigned grid = (unsigned)(((int64_t)ntiles * ((J.ntau + D - 1) / D) + WING_W - 1) / WING_W);
    if (few && P == 2) k_accum_fast<2, 2><<<grid, 32 * WING_W, 0, st>>>(J, ntiles);
    else if (few) k_accum_fast<2, 4><<<grid, 32 * WING_W, 0, st>>>(J, ntiles);
    else if (P == 2) k_accum_fast<WING_D, 2><<<grid, 32 * WING_W, 0, st>>>(J, ntiles);
    else k_accum_fast<WING_D, 4><<<grid, 32 * WING_W, 0, st>>>(J, ntiles);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

// the persistent wing pass over njobs jobs (device array), P wavelengths per lane; ctas counts CTAs of 16
// warps (two of the kernel's)
int fsg_launch_accum_batch(cudaStream_t st, int P, const WingJob *jobs, const int *item0, int njobs, int ctas,
                           unsigned *queue) {
    const size_t smem = WING_BW * (P == 2 ? sizeof(WingWarp<WING_D, 2>) : sizeof(WingWarp<WING_D, 4>));
    const unsigned grid = (unsigned)ctas * (16 / WING_BW);
    const void *fn = P == 2 ? (const void *)k_accum_batch<WING_D, 2> : (const void *)k_accum_batch<WING_D, 4>;
    if (cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem) != cudaSuccess) return FSG_E_CUDA;
    if (P == 2) k_accum_batch<WING_D, 2><<<grid, 32 * WING_BW, smem, st>>>(jobs, item0, njobs, queue);
    else k_accum_batch<WING_D, 4><<<grid, 32 * WING_BW, smem, st>>>(jobs, item0, njobs, queue);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

// Core pass.  Over each line's core range [cl, cr], the points where fl32(t) < 195.5 (s < 196): the
// table lerp or the continued fraction, as HVoigt branches (voigt.f90:81-107); the wing pass takes the
// others (the same FP32 test splits the points, so each is evaluated once).  A warp owns 32 wavelengths x
// CORE_D depths, Kahan sums in registers; warps share nothing.  It queues the lines whose core range meets
// the tile and stages them CORE_G at a time, double-buffered: the headers by plain loads, each line's records of the
// warp's depths by one bulk copy, a group's copies completing on the buffer's mbarrier (waits bounded; on
// expiry the kernel reports FSG_E_TIMEOUT, waits for its copies in flight, bounded again, and leaves).  Per
// line a lane forms its depths' branch predicates four at a time and issues their table gathers (one 16-byte
// load of the cell-major VgtTab copy each) together.
//
// What bounds it: instruction issue (60 to 70 % of the cycles) and the gathers, one 128-byte line of L1 a lane.  Hence
// floor() by an addition and not by conversions (the conversion unit takes 8 cycles a warp, the FP64 one 2), the
// continued fraction and whole depth groups left out where no lane needs them, and no barrier between depth groups.
// Against a CTA per tile that staged all depths of a chunk: 1e6 lines, 483,000 wavelengths, 56 depths 15.4 -> 11.5 ms; a
// batch of 24 atmospheres 19.7 -> 12.9 ms; 20,000 lines, 40,001 wavelengths 736 -> 500 us.  5 CTAs a SM (96
// registers): 4 take 7 % longer, 6 spill; the persistent form spills at 5.
//
// The segments' Kahan sums are added in FP64 (one sum over all classes of a long list is 3 % further from 64 bits: rms of
// LineOpac 5.2e-8 against 5.05e-8 for 50,000 molecular lines), in shared memory: added to LineOpac one by one they take
// 19.0 ms for those 1e6 lines.  Ten lines a group then, of one segment: 6 take 11.66 ms, 8 11.56, 10 11.48, 15 13.6 (less
// L1 for the gathers).  The two-depth form adds to LineOpac itself: 31 us for 300 lines, 37 through shared memory.
#define CORE_D 8                      // depths per warp (two groups of four gathers)
#define CORE_FEW 2                    // ... where there are few tiles
#define CORE_G 10                     // lines per group
#define CORE_GB 16                    // ... in the persistent form, which keeps no sums in shared memory
#define CORE_W 4                      // warps per CTA

template <int D, int G>
struct __align__(16) CoreWarp {
    CoreRec rec[2][G][D];
    LineHdr hdr[2][G];
    uint64_t bar[2];
    int queue[64];
};

template <class S_>
__device__ __forceinline__ void core_bars_init(S_ &S, int lane) {
    if (lane == 0) {
        mbar_init(&S.bar[0], 1);
        mbar_init(&S.bar[1], 1);
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
}

// One tile and depth group (depths t0 .. t0 + D - 1) of one job, by one warp with its mbarriers
// initialised; kk counts the groups of lines the warp has staged (their buffer and phase parity) across calls.
// PER_SEG: each segment's Kahan sums are added up in FP64, in tot (shared memory, [D][32]; null: LineOpac itself);
// otherwise one Kahan sum runs over all segments.  Returns false after a copy did not complete within its bound (error
// in *err).
template <bool PER_SEG, int D, int G>
__device__ __forceinline__ bool core_tile(const CoreJob &J, int tile, int t0, const float4 *__restrict__ vtab4, CoreWarp<D, G> &S,
                                          double (*tot)[32], int lane, unsigned &kk, int *err) {
    static_assert(2 * G <= 32, "a lane fills one line's padding");
    constexpr bool TOT = PER_SEG && D > CORE_FEW;
    constexpr int E = D < 4 ? D : 4;               // depths at a time
    const int ntau = J.ntau, nwl = J.nwl, nd = min(D, ntau - t0);
    bool any = false;                              // some segment has core ranges touching the tile
    for (int sg = 0; sg < J.nseg; sg++)
        any = any || J.tile_lo[sg * J.seg_stride + tile] <= J.tile_hi[sg * J.seg_stride + tile];
    if (!any) return true;
    const int p = tile * 32 + lane, p1 = p + 1;
    const int tile_first = tile * 32 + 1, tile_last = min(tile * 32 + 32, nwl);
    const double wd = J.wave[min(p, nwl - 1)];
    const float wvh = (float)wd, wvl = (float)(wd - (double)wvh);
    float sum[D], cmp[D];
#pragma unroll
    for (int d = 0; d < D; d++) {
        sum[d] = 0.0f;
        cmp[d] = 0.0f;
        if (TOT) tot[d][lane] = 0.0;
    }
    unsigned cnt = 0;
    // records past the last depth: none of their points is a core point (the copies leave them as they are).  A later
    // tile of the warp may have more depths there: its copies, of the async proxy, come after these stores
    if (nd < D) {
        if (lane < G * 2)
            for (int d = nd; d < D; d++) {
                CoreRec z{};
                z.c2m1 = 3.0e38f;
                (&S.rec[0][0][0])[lane * D + d] = z;
            }
        fence_proxy_async_shared();
    }
    auto work = [&](int b, int n) {
        for (int q = 0; q < n; q++) {
            const LineHdr h = S.hdr[b][q];
            const float dl = (wvh - h.wlh) + (wvl - h.wll);
            // the wing pass's x: the same branch split; outside the core range nothing is below 195.5
            const float x = p1 >= h.cl && p1 <= h.cr ? dl * dl : 3.0e38f;
            const double adl = fabs(wd - ((double)h.wlh + (double)h.wll)), adl125 = adl * 125.0;
            const CoreRec *__restrict__ rec = S.rec[b][q];
#pragma unroll
            for (int g0 = 0; g0 < D; g0 += E) {
                bool core[E], tab[E], some = false, cf = false;
#pragma unroll
                for (int e = 0; e < E; e++) {
                    core[e] = fmaf(x, rec[g0 + e].vv2, rec[g0 + e].c2m1) < 195.5f;
                    some = some || core[e];
                }
                if (!__any_sync(0xffffffffu, some)) continue;
                float tv[E];
                float4 gv[E];
#pragma unroll
                for (int e = 0; e < E; e++) {
                    // column and fraction: 2^52 added towards minus infinity leaves floor(v / 0.008) in the low word
                    const double fv = adl125 * rec[g0 + e].vv, m = __dadd_rd(fv, 4503599627370496.0);
                    const int iv = __double2loint(m), ia = rec[g0 + e].ia;
                    tab[e] = core[e] && iv < FSG_NVV - 1 && ia > 0;
                    cf = cf || (core[e] && !tab[e]);
                    tv[e] = (float)(fv - (m - 4503599627370496.0));
                    if (tab[e]) gv[e] = __ldg(vtab4 + ((ia - 1) * FSG_NV1 + iv));
                }
                cf = __any_sync(0xffffffffu, cf);
#pragma unroll
                for (int e = 0; e < E; e++) {
                    const CoreRec &cr = rec[g0 + e];
                    const float c0 = gv[e].x + tv[e] * (gv[e].y - gv[e].x), c1 = gv[e].z + tv[e] * (gv[e].w - gv[e].z);
                    const float h = c0 + cr.ua * (c1 - c0);
                    float y = fmaf(h, cr.cop, -cmp[g0 + e]);     // the Kahan step takes the product unrounded
                    if (cf) {
                        const float w = hv_cf32((float)(adl * cr.vv), cr.a);
                        const float yc = fmaf(w, cr.cop, -cmp[g0 + e]);
                        y = tab[e] ? y : yc;
                    }
                    if (core[e]) {
                        const float t = sum[g0 + e] + y;
                        cmp[g0 + e] = (t - sum[g0 + e]) - y;
                        sum[g0 + e] = t;
                        cnt++;
                    }
                }
            }
        }
    };
    const unsigned bytes = (unsigned)(nd * (int)sizeof(CoreRec));
    double *dst = J.lineopac + (size_t)p * ntau + t0;
    int head = 0, ncand = 0, sg = 0, base = 0, hi = -1, nprev = 0;
    const unsigned kk0 = kk;
    bool ok = true;
    for (;;) {
        bool cut = false;                              // the group in flight is the last of its segment
        while (ncand < G) {                            // lines into the queue
            if (base > hi) {
                if (sg == J.nseg || (PER_SEG && ncand)) break;     // no group of two segments
                base = J.tile_lo[sg * J.seg_stride + tile];
                hi = J.tile_hi[sg * J.seg_stride + tile];
                sg++;
                cut = true;
                continue;
            }
            const int i = base + lane;
            bool sel = false;
            if (i <= hi) {
                const int2 c = *(const int2 *)&J.hdr[i].cl;
                sel = c.x <= c.y && c.y >= tile_first && c.x <= tile_last;
            }
            base += 32;
            const unsigned m = __ballot_sync(0xffffffffu, sel);
            if (sel) S.queue[(head + ncand + __popc(m & ((1u << lane) - 1u))) & 63] = i;
            ncand += __popc(m);
        }
        __syncwarp();                                   // the queue is written, and the buffer's last group done with
        const int n = min(ncand, G), b = kk & 1;
        if (n) {                                        // a group into flight
            if (lane == 0) mbar_expect_tx(&S.bar[b], n * bytes + J.extra_tx);
            __syncwarp();
            if (lane < n) {
                const int i = S.queue[(head + lane) & 63];
                tma_bulk_g2s(S.rec[b][lane], J.core + (size_t)i * ntau + t0, bytes, &S.bar[b]);
                S.hdr[b][lane] = J.hdr[i];
            }
            head += n;
            ncand -= n;
            kk++;
        }
        if (nprev) {                                    // the group before: staged as number g
            const unsigned g = kk - (n ? 2 : 1);
            ok = __all_sync(0xffffffffu, mbar_wait(&S.bar[g & 1], (g >> 1) & 1, J.wait_ns));
            if (!ok) break;
            work(g & 1, nprev);
            // (the last sums are added here too: with a copy of this behind the loop the sparse tiles of a batch took 0.27 ms
            // for 0.20)
            if ((PER_SEG && cut) || !n) {
#pragma unroll
                for (int d = 0; d < D; d++) {
                    const double v = (double)sum[d] - (double)cmp[d];
                    if (TOT) tot[d][lane] += v;
                    else if (p < nwl && d < nd) dst[d] += v;
                    sum[d] = 0.0f;
                    cmp[d] = 0.0f;
                }
            }
        }
        nprev = n;
        if (!n) break;                                  // nothing in flight and no line left
    }
    if (TOT && ok && kk != kk0 && p < nwl) {            // some line has points here
#pragma unroll
        for (int d = 0; d < D; d++)
            if (d < nd) dst[d] += tot[d][lane];
    }
    if (!ok) {
        if (lane == 0) {
            atomicExch(err, FSG_E_TIMEOUT);
            for (unsigned g = kk - 2; g != kk; g++) mbar_wait(&S.bar[g & 1], (g >> 1) & 1, J.wait_ns);
        }
        __syncwarp();
        return false;
    }
    if (J.nevals) {
        unsigned long long v = cnt;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0 && v) atomicAdd(J.nevals, v);
    }
    return true;
}

// one (tile, depth group) per warp, the groups of a tile in turn
template <int D>
__global__ void __launch_bounds__(32 * CORE_W, 5)
k_core_fast(CoreJob J, int ntiles, const float4 *__restrict__ vtab4, int *__restrict__ err) {
    __shared__ CoreWarp<D, CORE_G> S[CORE_W];
    __shared__ double tot_s[D > CORE_FEW ? CORE_W : 1][D][32];
    double (*tot)[32] = D > CORE_FEW ? tot_s[threadIdx.x >> 5] : nullptr;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, ng = (J.ntau + D - 1) / D;
    const int64_t item = (int64_t)blockIdx.x * CORE_W + warp;
    if (item >= (int64_t)ntiles * ng) return;           // warps are independent: no CTA barrier
    core_bars_init(S[warp], lane);
    unsigned kk = 0;
    core_tile<true>(J, (int)(item / ng), (int)(item % ng) * D, vtab4, S[warp], tot, lane, kk, err);
}

// persistent form: warps take (job, tile, depth group) items from the queue
__global__ void __launch_bounds__(32 * CORE_W, 4)
k_core_batch(const CoreJob *__restrict__ jobs, const int *__restrict__ item0, int njobs,
             const float4 *__restrict__ vtab4, unsigned *queue, int *__restrict__ err) {
    __shared__ CoreWarp<CORE_D, CORE_GB> S[CORE_W];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    core_bars_init(S[warp], lane);
    unsigned kk = 0;
    const int total = item0[njobs];
    for (;;) {
        int item = 0;
        if (lane == 0) item = (int)atomicAdd(queue, 1u);
        item = __shfl_sync(0xffffffffu, item, 0);
        if (item >= total) break;
        int a = 0, b = njobs - 1;                          // job with item0[a] <= item < item0[a + 1]
        while (a < b) { int m = (a + b + 1) >> 1; if (item0[m] <= item) a = m; else b = m - 1; }
        const CoreJob J = jobs[a];
        const int ng = fsg_core_groups(J.ntau), r = item - item0[a];
        if (!core_tile<false>(J, r / ng, (r % ng) * CORE_D, vtab4, S[warp], nullptr, lane, kk, err)) break;
    }
}

int fsg_launch_core_fast(cudaStream_t st, const CoreJob &J, const float4 *vtab4, int *err) {
    const int ntiles = (J.nwl + 31) / 32;
    const int D = few_tiles(ntiles, J.ntau) ? CORE_FEW : CORE_D;
    const unsigned grid = (unsigned)(((int64_t)ntiles * ((J.ntau + D - 1) / D) + CORE_W - 1) / CORE_W);
    if (D == CORE_FEW) k_core_fast<CORE_FEW><<<grid, 32 * CORE_W, 0, st>>>(J, ntiles, vtab4, err);
    else k_core_fast<CORE_D><<<grid, 32 * CORE_W, 0, st>>>(J, ntiles, vtab4, err);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

// the persistent core pass over njobs jobs (device array) of at most ntau_max depths; ctas counts CTAs of one
// warp per depth group
int fsg_launch_core_batch(cudaStream_t st, int ntau_max, const CoreJob *jobs, const int *item0, int njobs,
                          int ctas, const float4 *vtab4, unsigned *queue, int *err) {
    const int64_t warps = (int64_t)ctas * fsg_core_groups(ntau_max);
    k_core_batch<<<(unsigned)((warps + CORE_W - 1) / CORE_W), 32 * CORE_W, 0, st>>>(jobs, item0, njobs, vtab4, queue, err);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

__global__ void k_tile_reset(int ntiles, int *lo, int *hi) {
    int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < ntiles) { lo[i] = 0x7fffffff; hi[i] = -1; }
}

// ---- tile candidate ranges of one block: lo/hi of the block-local line index -------------------
// The block's lines are in wavelength order.  With R_j = max_{i<=j} right_i (prefix max) and
// S_j = min_{i>=j} left_i (suffix min), both non-decreasing in j, the lines whose span [left,
// right] meets tile [f, l] all lie in [lo, hi] with lo = first j with R_j >= f and hi = last j
// with S_j <= l; both come from one binary search per tile.  Spans are the windows (use_core = 0)
// or the core ranges (use_core = 1; lines without one are left out).
__device__ __forceinline__ void span_of(const LineHdr &h, int use_core, int *l, int *r) {
    int a = use_core ? h.cl : h.ileft, b = use_core ? h.cr : h.iright;
    if (a > b) { a = 0x7fffffff; b = -1; }
    *l = a; *r = b;
}

// right_j in order, left_j in reverse order (rev[k] = left_{nb-1-k})
__global__ void k_span_extract(int nb, int use_core, const LineHdr *__restrict__ hdr, int *right, int *rev_left) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nb) return;
    int l, r;
    span_of(hdr[j], use_core, &l, &r);
    right[j] = r;
    rev_left[nb - 1 - j] = l;
}

// R: prefix max of right (non-decreasing); V: prefix min of reversed left, S_j = V[nb-1-j]
__global__ void k_tile_search(int nb, int ntiles, int tw, int nwl, const int *__restrict__ R,
                              const int *__restrict__ V, int *lo, int *hi) {
    int t = blockIdx.x * blockDim.x + threadIdx.x;
    if (t >= ntiles) return;
    const int f = t * tw + 1, l = min(t * tw + tw, nwl);
    int a = 0, b = nb;                                   // first j with R_j >= f
    while (a < b) { int m = (a + b) >> 1; if (R[m] >= f) b = m; else a = m + 1; }
    const int jlo = a;
    a = 0; b = nb;                                       // first j with S_j > l
    while (a < b) { int m = (a + b) >> 1; if (V[nb - 1 - m] > l) b = m; else a = m + 1; }
    lo[t] = jlo;
    hi[t] = a - 1;
}

// tile count of the narrowest tiles (sizes the lo/hi arrays)
int fsg_fast_tiles(int nwl) { return (nwl + 31) / 32; }

// scratch bytes of fsg_launch_tile_span for nb lines
size_t fsg_tile_span_scratch(int64_t nb) {
    size_t t1 = 0, t2 = 0;
    cub::DeviceScan::InclusiveScan(nullptr, t1, (const int *)nullptr, (int *)nullptr, cuda::maximum<>{}, (int)nb);
    cub::DeviceScan::InclusiveScan(nullptr, t2, (const int *)nullptr, (int *)nullptr, cuda::minimum<>{}, (int)nb);
    return 4 * sizeof(int) * (size_t)nb + std::max(t1, t2) + 256;
}

int fsg_launch_tile_span_tw(cudaStream_t s, int tw, int use_core, int nwl, int64_t nb, const LineHdr *hdr, int *lo,
                            int *hi, void *scratch, size_t scratch_bytes);

int fsg_launch_tile_span(cudaStream_t s, int cls, int nwl, int64_t nb, const LineHdr *hdr, int *lo, int *hi,
                         void *scratch, size_t scratch_bytes) {
    return fsg_launch_tile_span_tw(s, cls < 0 ? 32 : 32 * fsg_class_pix(cls), cls < 0 ? 1 : 0, nwl, nb, hdr, lo, hi,
                                   scratch, scratch_bytes);
}

// as k_span_extract, over the windows of FP64 headers
__global__ void k_span_extract64(int nb, const LineHdr64 *__restrict__ hdr, int *right, int *rev_left) {
    int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nb) return;
    int l = hdr[j].il, r = hdr[j].ir;
    if (l > r) { l = 0x7fffffff; r = -1; }
    right[j] = r;
    rev_left[nb - 1 - j] = l;
}

// scans of the extracted spans, then one binary search per tile; scratch: fsg_tile_span_scratch(nb) bytes,
// its first 2 nb ints the spans
static int tile_search(cudaStream_t s, int tw, int nwl, int64_t nb, int *lo, int *hi, void *scratch,
                       size_t scratch_bytes) {
    const int ntiles = (nwl + tw - 1) / tw;
    int *right = (int *)scratch, *revl = right + nb, *R = revl + nb, *V = R + nb;
    void *tmp = (void *)(((uintptr_t)(V + nb) + 255) & ~(uintptr_t)255);
    size_t tb = scratch_bytes - ((char *)tmp - (char *)scratch);
    if (cub::DeviceScan::InclusiveScan(tmp, tb, right, R, cuda::maximum<>{}, (int)nb, s) != cudaSuccess) return FSG_E_CUDA;
    if (cub::DeviceScan::InclusiveScan(tmp, tb, revl, V, cuda::minimum<>{}, (int)nb, s) != cudaSuccess) return FSG_E_CUDA;
    k_tile_search<<<(ntiles + 255) / 256, 256, 0, s>>>((int)nb, ntiles, tw, nwl, R, V, lo, hi);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

// tile ranges for tiles of tw wavelengths over the windows (use_core = 0) or the core ranges
int fsg_launch_tile_span_tw(cudaStream_t s, int tw, int use_core, int nwl, int64_t nb, const LineHdr *hdr, int *lo,
                            int *hi, void *scratch, size_t scratch_bytes) {
    const int ntiles = (nwl + tw - 1) / tw;
    if (nb <= 0) {
        k_tile_reset<<<(ntiles + 255) / 256, 256, 0, s>>>(ntiles, lo, hi);
        return FSG_OK;
    }
    int *right = (int *)scratch, *revl = right + nb;
    k_span_extract<<<(unsigned)((nb + 255) / 256), 256, 0, s>>>((int)nb, use_core, hdr, right, revl);
    return tile_search(s, tw, nwl, nb, lo, hi, scratch, scratch_bytes);
}

// the same over the windows of FP64 headers (nb > 0)
int fsg_launch_tile_span64(cudaStream_t s, int tw, int nwl, int64_t nb, const LineHdr64 *hdr, int *lo, int *hi,
                           void *scratch, size_t scratch_bytes) {
    int *right = (int *)scratch, *revl = right + nb;
    k_span_extract64<<<(unsigned)((nb + 255) / 256), 256, 0, s>>>((int)nb, hdr, right, revl);
    return tile_search(s, tw, nwl, nb, lo, hi, scratch, scratch_bytes);
}

// Restriction to the wavelength range [i0, i1]: lines whose window misses it are marked weak for the
// selection, the others keep their flags and get the window clipped to the range.
__global__ void k_range_clip(int64_t n, const int32_t *fl, const int32_t *il, const int32_t *ir, int i0, int i1,
                             int32_t *rf, int32_t *rl, int32_t *rr) {
    int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    int f = fl[i], a = max(il[i], i0), b = min(ir[i], i1);
    if (a > b) f |= FSG_F_WEAK;
    rf[i] = f; rl[i] = a; rr[i] = b;
}

void fsg_launch_range_clip(cudaStream_t s, int64_t n, const int32_t *fl, const int32_t *il, const int32_t *ir, int i0,
                           int i1, int32_t *rf, int32_t *rl, int32_t *rr) {
    if (n > 0) k_range_clip<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, fl, il, ir, i0, i1, rf, rl, rr);
}

// ---- window-width classes and order-preserving compaction -----------------------------------
// class 0: windows up to 256 wavelengths; class c: up to 256 * 2^c.
__device__ __forceinline__ int width_class(int il, int ir) {
    int w = ir - il + 1;
    int c = 0;
    while ((CLASS_W0 << (c + 1)) < w && c < 30) c++;
    return c;
}

#define SCAN_BS 1024
// selection predicate: cls >= 0 retained lines of that width class (He I shifted lines excluded),
// -1 every retained line, -2 retained wide lines (flag bit 3), -3 retained He I shifted lines
__device__ __forceinline__ int sel_pred(int f, int il, int ir, int cls) {
    if (f & FSG_F_WEAK) return 0;
    if (cls == -1) return 1;
    if (cls == -2) return (f & FSG_F_WIDE) != 0;
    if (cls == -3) return ((f >> 8) & 255) != 0;         // He I lines with Stark-shifted profiles
    if ((f >> 8) & 255) return 0;                        // ... which the FP32 classes leave out
    return width_class(il, ir) == cls;
}
// Count retained lines of class `cls` (cls < 0: every retained line) per CTA of SCAN_BS lines.
__global__ void k_sel_count(int64_t n, const int32_t *flags, const int32_t *il, const int32_t *ir, int cls,
                            int *counts) {
    __shared__ int warp_sums[SCAN_BS / 32];
    int64_t i = (int64_t)blockIdx.x * SCAN_BS + threadIdx.x;
    int pred = 0;
    if (i < n) pred = sel_pred(flags[i], il[i], ir[i], cls);
    unsigned m = __ballot_sync(0xffffffffu, pred);
    if ((threadIdx.x & 31) == 0) warp_sums[threadIdx.x >> 5] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int w = 0; w < SCAN_BS / 32; w++) s += warp_sums[w];
        counts[blockIdx.x] = s;
    }
}

// Exclusive scan of the per-CTA counts (single CTA, serial over chunks of 1024).
__global__ void k_scan_counts(int nblk, const int *counts, int64_t *offs, int64_t *total) {
    __shared__ int64_t buf[1024];
    __shared__ int64_t carry;
    if (threadIdx.x == 0) carry = 0;
    __syncthreads();
    for (int base = 0; base < nblk; base += 1024) {
        int i = base + threadIdx.x;
        int64_t v = (i < nblk) ? counts[i] : 0;
        buf[threadIdx.x] = v;
        __syncthreads();
        for (int off = 1; off < 1024; off <<= 1) {
            int64_t t = (threadIdx.x >= off) ? buf[threadIdx.x - off] : 0;
            __syncthreads();
            buf[threadIdx.x] += t;
            __syncthreads();
        }
        if (i < nblk) offs[i] = carry + buf[threadIdx.x] - v;
        __syncthreads();
        if (threadIdx.x == 1023) carry += buf[1023];
        __syncthreads();
    }
    if (threadIdx.x == 0) *total = carry;
}

__global__ void k_sel_scatter(int64_t n, const int32_t *flags, const int32_t *il, const int32_t *ir, int cls,
                              const int64_t *offs, int64_t *out) {
    __shared__ int warp_offs[SCAN_BS / 32];
    int64_t i = (int64_t)blockIdx.x * SCAN_BS + threadIdx.x;
    int pred = 0;
    if (i < n) pred = sel_pred(flags[i], il[i], ir[i], cls);
    unsigned m = __ballot_sync(0xffffffffu, pred);
    int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    if (lane == 0) warp_offs[w] = __popc(m);
    __syncthreads();
    if (threadIdx.x == 0) {
        int s = 0;
        for (int q = 0; q < SCAN_BS / 32; q++) { int t = warp_offs[q]; warp_offs[q] = s; s += t; }
    }
    __syncthreads();
    if (pred) {
        int r = warp_offs[w] + __popc(m & ((1u << lane) - 1u));
        out[offs[blockIdx.x] + r] = i;
    }
}

// Select (in order) the retained lines of class cls into out[]; *count receives the number (device).
int fsg_select(cudaStream_t s, int64_t n, const int32_t *flags, const int32_t *il, const int32_t *ir, int cls,
               int *counts, int64_t *offs, int64_t *out, int64_t *d_total) {
    if (n <= 0) { cudaMemsetAsync(d_total, 0, sizeof(int64_t), s); return FSG_OK; }
    int nblk = (int)((n + SCAN_BS - 1) / SCAN_BS);
    k_sel_count<<<nblk, SCAN_BS, 0, s>>>(n, flags, il, ir, cls, counts);
    k_scan_counts<<<1, 1024, 0, s>>>(nblk, counts, offs, d_total);
    k_sel_scatter<<<nblk, SCAN_BS, 0, s>>>(n, flags, il, ir, cls, offs, out);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

// Histogram of window classes of the retained lines (for the host loop over classes).  Counted in shared memory: one
// global addition per line on a few addresses took 3.6 ms for 1e7 lines, a CTA's share at a time 47 us.
__global__ void __launch_bounds__(256) k_class_hist(int64_t n, const int32_t *__restrict__ flags, const int32_t *__restrict__ il,
                                                    const int32_t *__restrict__ ir, unsigned long long *hist) {
    __shared__ unsigned h[32];
    if (threadIdx.x < 32) h[threadIdx.x] = 0u;
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * 256 + threadIdx.x; i < n; i += (int64_t)gridDim.x * 256) {
        const int f = flags[i];
        if (!(f & FSG_F_WEAK) && !((f >> 8) & 255)) atomicAdd(&h[width_class(il[i], ir[i])], 1u);
    }
    __syncthreads();
    if (threadIdx.x < 32 && h[threadIdx.x]) atomicAdd(&hist[threadIdx.x], (unsigned long long)h[threadIdx.x]);
}

void fsg_launch_class_hist(cudaStream_t s, int64_t n, const int32_t *flags, const int32_t *il,
                           const int32_t *ir, unsigned long long *hist) {
    if (n > 0) k_class_hist<<<(unsigned)std::min<int64_t>((n + 255) / 256, 148 * 8), 256, 0, s>>>(n, flags, il, ir, hist);
}

// Motype 1 is folded into the records; nothing else to finish.

int fsg_select_wide(cudaStream_t s, int64_t n, const int32_t *flags, int *counts, int64_t *offs, int64_t *out,
                    int64_t *d_total) {
    return fsg_select(s, n, flags, flags, flags, -2, counts, offs, out, d_total);
}

// ---- records in window-width-class order -------------------------------------------------------
// A list that fits one block (an atmosphere of a batch, or a single synthesis) is one record array, grouped by window-width
// class (retained lines of class 0, 1, ..., ncls - 1, then the rejected ones), in list (wavelength)
// order inside each class.  A tile's candidate range is then searched inside one class, so it spans
// lines of like width only: the prefix-max / suffix-min spans of a single list with a few very wide
// windows would stage every line between such a window's centre and the tile.
#define BCLS_MAX 24

// class of a line for the record order: ncls for rejected lines, empty windows and He I lines with a Stark shift
// per depth (which the FP32 classes leave out)
__device__ __forceinline__ int bclass_of(int f, int il, int ir, int ncls) {
    if ((f & FSG_F_WEAK) || il > ir || ((f >> 8) & 255)) return ncls;
    return min(width_class(il, ir), ncls - 1);
}

// lines per class and CTA of SCAN_BS lines: counts[c * nblk + blk], c = 0 .. ncls
__global__ void k_bclass_count(int64_t n, const int32_t *__restrict__ flags, const int32_t *__restrict__ il,
                               const int32_t *__restrict__ ir, int ncls, int *counts) {
    __shared__ int h[BCLS_MAX + 1];
    for (int c = threadIdx.x; c <= ncls; c += blockDim.x) h[c] = 0;
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * SCAN_BS + threadIdx.x;
    if (i < n) atomicAdd(&h[bclass_of(flags[i], il[i], ir[i], ncls)], 1);
    __syncthreads();
    for (int c = threadIdx.x; c <= ncls; c += blockDim.x) counts[c * gridDim.x + blockIdx.x] = h[c];
}

// order[offs[c * nblk + blk] + rank of line i among the CTA's class-c lines] = i (stable)
__global__ void k_bclass_scatter(int64_t n, const int32_t *__restrict__ flags, const int32_t *__restrict__ il,
                                 const int32_t *__restrict__ ir, int ncls, const int64_t *__restrict__ offs,
                                 int64_t *order) {
    __shared__ int wc[SCAN_BS / 32][BCLS_MAX + 1];       // per warp and class: count, then prefix over warps
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    for (int k = threadIdx.x; k < (SCAN_BS / 32) * (BCLS_MAX + 1); k += blockDim.x) (&wc[0][0])[k] = 0;
    __syncthreads();
    const int64_t i = (int64_t)blockIdx.x * SCAN_BS + threadIdx.x;
    const int c = i < n ? bclass_of(flags[i], il[i], ir[i], ncls) : -1;
    const unsigned same = __match_any_sync(0xffffffffu, c);
    const int rank = __popc(same & ((1u << lane) - 1u));
    if (c >= 0 && rank == 0) wc[w][c] = __popc(same);  // the class's lowest lane in the warp
    __syncthreads();
    if (threadIdx.x <= ncls) {
        int acc = 0;
        for (int q = 0; q < SCAN_BS / 32; q++) { const int t = wc[q][threadIdx.x]; wc[q][threadIdx.x] = acc; acc += t; }
    }
    __syncthreads();
    if (c >= 0) order[offs[c * gridDim.x + blockIdx.x] + wc[w][c] + rank] = i;
}

// Class order of n lines (ncls <= BCLS_MAX classes + the rejected): order[n] and the class offsets,
// class c starting at record offs[c * nblk] (nblk = ceil(n / SCAN_BS)); counts and offs hold
// (ncls + 1) * nblk entries.
int fsg_launch_bclass_order(cudaStream_t s, int64_t n, const int32_t *flags, const int32_t *il, const int32_t *ir,
                            int ncls, int *counts, int64_t *offs, int64_t *total, int64_t *order) {
    if (n <= 0 || ncls < 1 || ncls > BCLS_MAX) return n <= 0 ? FSG_OK : FSG_E_ARG;
    const int nblk = (int)((n + SCAN_BS - 1) / SCAN_BS);
    k_bclass_count<<<nblk, SCAN_BS, 0, s>>>(n, flags, il, ir, ncls, counts);
    k_scan_counts<<<1, 1024, 0, s>>>((ncls + 1) * nblk, counts, offs, total);
    k_bclass_scatter<<<nblk, SCAN_BS, 0, s>>>(n, flags, il, ir, ncls, offs, order);
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

// classes of an atmosphere's order: every window fits the grid, so the widest class is that of nwl
int fsg_bclass_count(int nwl) {
    int c = 0;
    while ((CLASS_W0 << (c + 1)) < nwl && c < 30) c++;
    return std::min(c + 1, BCLS_MAX);
}

// Segmented spans of the wing pass (windows) and of the core pass (core ranges) in one array of 2 nb keys,
// the core's after the wing's: key = (pass * BCLS_PASS + class) << 32 | value, so one prefix max (of right + 1)
// and one suffix min (of left) over the whole array stay inside each pass and class, and both key arrays are
// sorted.
#define BCLS_PASS 32
__global__ void k_bspan_extract(int nb, const LineHdr *__restrict__ hdr, const int64_t *__restrict__ offs, int nblk,
                                int ncls, unsigned long long *right, unsigned long long *rev_left) {
    const int j = blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nb) return;
    int seg = 0;
    while (seg < ncls && offs[(size_t)(seg + 1) * nblk] <= j) seg++;
    const LineHdr h = hdr[j];
    for (int pass = 0; pass < 2; pass++) {
        int l, r;
        span_of(h, pass, &l, &r);
        if (seg == ncls) { l = 0x7fffffff; r = -1; }
        const unsigned long long key = (unsigned long long)(pass * BCLS_PASS + seg) << 32;
        right[pass * nb + j] = key | (unsigned)(r + 1);
        rev_left[2 * nb - 1 - (pass * nb + j)] = key | (unsigned)l;
    }
}

// Tile t of class c (blockIdx.y) of the wing pass (blockIdx.z = 0: tiles of tw_n wavelengths for classes <=
// cnarrow, tw_w for the others) or the core pass (1: tiles of 32); lo/hi at c * stride + t are record indices of
// class c (lo > hi: no line touches it).
struct SpanOut { int *lo, *hi, stride; };
__global__ void k_btile_search(int nb, int cnarrow, int tw_n, int tw_w, int nwl,
                               const unsigned long long *__restrict__ R, const unsigned long long *__restrict__ V,
                               SpanOut wing, SpanOut core) {
    const int t = blockIdx.x * blockDim.x + threadIdx.x, c = blockIdx.y, pass = blockIdx.z;
    const int tw = pass ? 32 : c <= cnarrow ? tw_n : tw_w;
    if (t >= (nwl + tw - 1) / tw) return;
    const SpanOut out = pass ? core : wing;
    const int f = t * tw + 1, l = min(t * tw + tw, nwl), n = 2 * nb;
    const unsigned long long key = (unsigned long long)(pass * BCLS_PASS + c) << 32;
    const unsigned long long kf = key | (unsigned)(f + 1), kl = key | (unsigned)l;
    int a = 0, b = n;                                    // first j with R_j >= kf
    while (a < b) { const int m = (a + b) >> 1; if (R[m] >= kf) b = m; else a = m + 1; }
    const int jlo = a;
    a = 0; b = n;                                        // first j with S_j > kl, S_j = V[n - 1 - j]
    while (a < b) { const int m = (a + b) >> 1; if (V[n - 1 - m] > kl) b = m; else a = m + 1; }
    out.lo[c * out.stride + t] = jlo - pass * nb;
    out.hi[c * out.stride + t] = a - 1 - pass * nb;
}

size_t fsg_bspan_scratch(int64_t nb) {
    size_t t1 = 0, t2 = 0;
    typedef unsigned long long u64;
    const int n = (int)(2 * nb);
    cub::DeviceScan::InclusiveScan(nullptr, t1, (const u64 *)nullptr, (u64 *)nullptr, cuda::maximum<>{}, n);
    cub::DeviceScan::InclusiveScan(nullptr, t2, (const u64 *)nullptr, (u64 *)nullptr, cuda::minimum<>{}, n);
    return 4 * sizeof(u64) * (size_t)n + std::max(t1, t2) + 256;
}

// tile ranges of every class of a class-ordered record array, both passes (offs: class c starts at record
// offs[c * nblk], as fsg_launch_bclass_order leaves them); wing and core arrays hold ncls rows of wstride /
// cstride entries
int fsg_launch_btile_span(cudaStream_t s, int64_t nb, const LineHdr *hdr, const int64_t *offs, int nblk, int ncls,
                          int cnarrow, int tw_n, int tw_w, int nwl, int wstride, int *wlo, int *whi, int cstride, int *clo,
                          int *chi, void *scratch, size_t scratch_bytes) {
    typedef unsigned long long u64;
    if (nb <= 0) {
        k_tile_reset<<<(wstride * ncls + 255) / 256, 256, 0, s>>>(wstride * ncls, wlo, whi);
        k_tile_reset<<<(cstride * ncls + 255) / 256, 256, 0, s>>>(cstride * ncls, clo, chi);
        return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
    }
    const int n = (int)(2 * nb);
    u64 *right = (u64 *)scratch, *revl = right + n, *R = revl + n, *V = R + n;
    void *tmp = (void *)(((uintptr_t)(V + n) + 255) & ~(uintptr_t)255);
    size_t tb = scratch_bytes - ((char *)tmp - (char *)scratch);
    k_bspan_extract<<<(unsigned)((nb + 255) / 256), 256, 0, s>>>((int)nb, hdr, offs, nblk, ncls, right, revl);
    if (cub::DeviceScan::InclusiveScan(tmp, tb, right, R, cuda::maximum<>{}, n, s) != cudaSuccess) return FSG_E_CUDA;
    if (cub::DeviceScan::InclusiveScan(tmp, tb, revl, V, cuda::minimum<>{}, n, s) != cudaSuccess) return FSG_E_CUDA;
    const int tmax = (nwl + 31) / 32;
    k_btile_search<<<dim3((tmax + 255) / 256, ncls, 2), 256, 0, s>>>((int)nb, cnarrow, tw_n, tw_w, nwl, R, V,
                                                                     SpanOut{ wlo, whi, wstride },
                                                                     SpanOut{ clo, chi, cstride });
    return cudaGetLastError() == cudaSuccess ? FSG_OK : FSG_E_CUDA;
}

// Gather the retained lines' SoA fields and per-line outputs into packed arrays (PACK,
// synth.f90:915-933).  buf must hold 64 bytes per packed line.
__global__ void k_gather_lines(LineView L, const int64_t *idx, int64_t nw, double *wl, float *elo, float *gf,
                               float *grad, float *gqst, float *gvdw, int32_t *spc, int32_t *ismol, int32_t *ihe,
                               const int32_t *f0, const int32_t *l0, const int32_t *r0, int32_t *f1, int32_t *l1,
                               int32_t *r1) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j >= nw) return;
    int64_t i = idx[j];
    wl[j] = L.wl[i]; elo[j] = L.elo[i]; gf[j] = L.gf[i]; grad[j] = L.grad[i]; gqst[j] = L.gqst[i];
    gvdw[j] = L.gvdw[i]; spc[j] = L.spc[i];
    if (L.ismol) ismol[j] = L.ismol[i];
    if (L.ihe) ihe[j] = L.ihe[i];
    f1[j] = f0[i]; l1[j] = l0[i]; r1[j] = r0[i];
}

void fsg_launch_gather_lines(cudaStream_t s, const LineView &L, const int64_t *idx, int64_t nw, char *buf,
                             const int32_t *f0, const int32_t *l0, const int32_t *r0, LineView *W, int32_t **f1,
                             int32_t **l1, int32_t **r1) {
    size_t n = (size_t)(nw > 0 ? nw : 1);
    double *wl = (double *)buf;
    float *elo = (float *)(wl + n), *gf = elo + n, *grad = gf + n, *gqst = grad + n, *gvdw = gqst + n;
    int32_t *spc = (int32_t *)(gvdw + n), *ismol = spc + n, *ihe = ismol + n, *ff = ihe + n, *ll = ff + n, *rr = ll + n;
    if (nw > 0)
        k_gather_lines<<<(unsigned)((nw + 255) / 256), 256, 0, s>>>(L, idx, nw, wl, elo, gf, grad, gqst, gvdw, spc,
                                                                    ismol, ihe, f0, l0, r0, ff, ll, rr);
    *W = L;
    W->n = nw; W->wl = wl; W->elo = elo; W->gf = gf; W->grad = grad; W->gqst = gqst; W->gvdw = gvdw; W->spc = spc;
    W->ismol = L.ismol ? ismol : nullptr; W->ihe = L.ihe ? ihe : nullptr;
    *f1 = ff; *l1 = ll; *r1 = rr;
}

__global__ void k_scatter_flags(int64_t nw, const int64_t *idx, const int32_t *pf, int32_t *flags) {
    int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (j < nw) flags[idx[j]] = pf[j];
}

void fsg_launch_scatter_flags(cudaStream_t s, int64_t nw, const int64_t *idx, const int32_t *pf, int32_t *flags) {
    if (nw > 0) k_scatter_flags<<<(unsigned)((nw + 255) / 256), 256, 0, s>>>(nw, idx, pf, flags);
}
