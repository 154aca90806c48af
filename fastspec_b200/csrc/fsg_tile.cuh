// fsg_tile.cuh -- the lines of one wavelength tile, picked by one warp
#pragma once
#include "fsg_internal.cuh"

__device__ __forceinline__ int2 window_of(const LineHdr &h) { return *(const int2 *)&h.ileft; }
__device__ __forceinline__ int2 window_of(const LineHdr64 &h) { return *(const int2 *)&h.il; }

// Rows lo .. hi whose windows meet the wavelengths first .. last, in order: group(head, n) gets them G at a
// time (the last call fewer) as queue[(head + i) & 63], i < n; queue holds 64 rows of the calling warp.
template <int G, class H, class F>
__device__ __forceinline__ void tile_lines(const H *__restrict__ hdr, int lo, int hi, int first, int last, int *queue,
                                           int lane, F group) {
    int head = 0, cnt = 0;
    const int2 none = make_int2(1, 0);
    int2 next = lo + lane <= hi ? window_of(hdr[lo + lane]) : none;
    for (int base = lo; base <= hi; base += 32) {
        const int j = base + lane;
        const int2 w = next;                            // the next 32 windows are on their way meanwhile
        next = j + 32 <= hi ? window_of(hdr[j + 32]) : none;
        const bool sel = w.x <= w.y && w.x <= last && w.y >= first;
        const unsigned m = __ballot_sync(0xffffffffu, sel);
        if (!m) continue;
        if (sel) queue[(head + cnt + __popc(m & ((1u << lane) - 1u))) & 63] = j;
        cnt += __popc(m);
        __syncwarp();
        while (cnt >= G) { group(head, G); head += G; cnt -= G; }
    }
    if (cnt > 0) group(head, cnt);
}
