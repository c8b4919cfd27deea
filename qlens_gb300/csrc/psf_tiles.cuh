// psf_tiles.cuh -- what the two builds by image tiles share, of the mixed path's X
// (k_psf_x, mixed.cu) and of the plain path's L' (k_psf64, psf.cu): the taps'
// table in shared memory and the list of (cell, tile) pairs that a footprint reaches.
#pragma once
#include "qlpix_internal.h"

namespace qlpix {

#define PSFX_R 8                        // rows of a tile (32 pixels wide)
#define PSFX_PAD_BYTES (96 * 1024)
__host__ __device__ __forceinline__ int psfx_pitch(int pny) { return (pny + 2 * PSFX_R - 2) | 1; }
static inline size_t psfx_taps(int pnx, int pny) { return (size_t)(pnx + 62) * psfx_pitch(pny); }

// The biased exponent of |x| (at least 1), 0 for zero, 2047 for infinities and NaN.
__device__ __forceinline__ int exponent_of(double x)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(x) << 1;
    return u == 0 ? 0 : max(1, (int)(u >> 53));
}

// The grid of a cell whose largest finite L has this biased exponent: that L times 2^shift
// lies in [1, 2) (a cell that sub-pixels only touch has none but small entries).
__device__ __forceinline__ int psf64_shift(int top) { return top ? 1023 - top : 0; }
// ... an entry's part in it
__device__ __forceinline__ int psf64_top(double v)
{
    const int e = exponent_of(v);
    return e == 2047 ? 0 : e;
}

// An entry of the plain path's columns: (image column, hi, lo, image row), L on the cell's
// grid 2^-(57 + shift) = hi 2^29 + lo (0 <= lo < 2^29, |hi| <= 2^29); infinities and NaN are
// marked by INT_MIN.
#define PSF64_BAD ((int)0x80000000)
__device__ __forceinline__ int4 psf64_entry(int i, int j, double v, int shift)
{
    const long long b = __double_as_longlong(v);
    const int e = (int)((b >> 52) & 0x7ff);
    if (e == 2047) return make_int4(i, PSF64_BAD, 0, j);
    const long long m = (b & 0xfffffffffffffll) | (e ? 1ll << 52 : 0);
    const int s = max(e, 1) - 1075 + 57 + shift;    // m 2^s, s <= 5
    const long long a = s >= 0 ? m << s : (s > -55 ? (m + (1ll << (-s - 1))) >> -s : 0);
    const long long q = b < 0 ? -a : a;
    return make_int4(i, (int)(q >> 29), (int)q & 0x1fffffff, j);
}

// ... and for FP64 sums, L's bits (low, high).
__device__ __forceinline__ int4 psf64_raw(int i, int j, double v)
{
    return make_int4(i, __double2loint(v), __double2hiint(v), j);
}

__device__ __forceinline__ int ent_col(int2 e) { return e.x >> 16; }
__device__ __forceinline__ int ent_row(int2 e) { return e.x & 0xffff; }
__device__ __forceinline__ int ent_col(int4 e) { return e.x; }
__device__ __forceinline__ int ent_row(int4 e) { return e.w; }

// The first of n entries sorted by image row whose row is at
// least jmin, by a whole warp: 32 probes a round.
template <typename E>
__device__ __forceinline__ int warp_lower_bound_row(const E* __restrict__ ent, int n, int jmin)
{
    const int lane = threadIdx.x & 31;
    int lo = 0, hi = n;                       // the answer lies in [lo, hi]
    while (hi - lo > 32) {
        const int step = (hi - lo + 31) / 32;
        const int p = lo + lane * step;
        const unsigned b = __ballot_sync(0xffffffffu, p >= hi || ent_row(ent[p]) >= jmin);
        if (b == 0) {
            lo = lo + 31 * step + 1;
        } else {
            const int f = __ffs(b) - 1;
            const int pf = lo + f * step;
            if (f > 0) lo = lo + (f - 1) * step + 1;
            hi = min(hi, pf);
        }
    }
    const int p = lo + lane;
    const unsigned b = __ballot_sync(0xffffffffu, p >= hi || ent_row(ent[p]) >= jmin);
    return b ? min(lo + __ffs(b) - 1, hi) : hi;
}

// The tiles that each cell's footprints reach: a warp per cell, its bitmap of the
// image's tiles in shared memory, span words at a time (one pass for images of up to
// 100 million pixels, 48 KB).
template <typename E>
__global__ void k_psfx_tiles(StaticData sd, const GridState* __restrict__ gs, const int* __restrict__ colptr,
                             const E* __restrict__ ent_g, int ntx, int nwords, int span,
                             const unsigned* __restrict__ active,
                             int* __restrict__ count, uint2* __restrict__ list)
{
    extern __shared__ unsigned mark_all[];
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, s = blockIdx.x * nw + (threadIdx.x >> 5);
    if (s >= gs->M) return;                                       // whole warps
    unsigned* mark = mark_all + (threadIdx.x >> 5) * span;
    const int pnx = sd.pnx, pny = sd.pny, nxh = pnx / 2, nyh = pny / 2;
    const int n = colptr[s + 1] - colptr[s];
    const E* ent = ent_g + colptr[s];
    for (int b0 = 0; b0 < nwords; b0 += span) {
        const int b1 = min(b0 + span, nwords);
        for (int i = lane; i < b1 - b0; i += 32) mark[i] = 0;
        __syncwarp();
        for (int e0 = 0; e0 < n; e0 += 32) {
            const E en = ent[min(e0 + lane, n - 1)];
            const int i0 = ent_col(en) - nxh, j0 = ent_row(en) - nyh;
            const int c0 = max(i0, 0) >> 5, c1 = (min(i0 + pnx, sd.nx) - 1) >> 5;
            const int t0 = max(j0, 0) / PSFX_R, t1 = (min(j0 + pny, sd.ny) - 1) / PSFX_R;
            // neighbours along a row mostly reach the same tiles: only the first marks them
            const bool same = __shfl_up_sync(0xffffffffu, c0, 1) == c0 & __shfl_up_sync(0xffffffffu, c1, 1) == c1 &
                              __shfl_up_sync(0xffffffffu, t0, 1) == t0 & __shfl_up_sync(0xffffffffu, t1, 1) == t1;
            if (lane > 0 && same) continue;
            for (int t = t0; t <= t1; t++) {
                const int k0 = t * ntx + c0, k1 = t * ntx + c1;
                for (int w = max(k0 >> 5, b0); w <= min(k1 >> 5, b1 - 1); w++) {
                    unsigned m = 0xffffffffu;
                    if (w == k0 >> 5) m &= 0xffffffffu << (k0 & 31);
                    if (w == k1 >> 5) m &= 0xffffffffu >> (31 - (k1 & 31));
                    if ((mark[w - b0] & m) != m) atomicOr(&mark[w - b0], m);
                }
            }
        }
        __syncwarp();
        for (int w0 = b0; w0 < b1; w0 += 32) {
            const int wd = w0 + lane;
            unsigned bits = wd < b1 ? mark[wd - b0] & active[wd] : 0u;
            int at = __popc(bits);
            for (int o = 1; o < 32; o <<= 1) {
                const int v = __shfl_up_sync(0xffffffffu, at, o);
                if (lane >= o) at += v;
            }
            const int total = __shfl_sync(0xffffffffu, at, 31);
            if (total == 0) continue;
            int base = 0;
            if (lane == 0) base = atomicAdd(count, total);
            at += __shfl_sync(0xffffffffu, base, 0) - __popc(bits);
            for (; bits; bits &= bits - 1) list[at++] = make_uint2(s, 32 * wd + __ffs(bits) - 1);
        }
        __syncwarp();
    }
}

}  // namespace qlpix
