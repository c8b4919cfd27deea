// mixed.cu -- mixed-precision inversion: tensor-core SYRK of F16 hi + lo parts,
// FP32 Cholesky of F and R, FP64 log det accumulation and FP64 iterative
// refinement of the source amplitudes.
//
//   X      = (P L sqrt(C^-1))^T by image tiles (exact fixed-point
//            sums), split into F16 hi + lo                       k_psf_x
//   F32    = X X^T on tcgen05 (block-sparse over pixel blocks)   k_syrk_tc
//   F32   += lambda R, R32 = R                                  k_reg32
//   L_F L_F^T = F32, L_R L_R^T = R32 (FP32 blocked Cholesky)    chol128.cuh
//   log det F, log det R: 2 sum log diag, accumulated in FP64
//   D = L^T P^T (C^-1 d)                     (FP64; L^T from L by source cell)
//   s = F32^-1 D, then `refine` times: r = D - L^T P^T C^-1 P L s - lambda R s (FP64),
//                                       s += F32^-1 r
//   model = P L s                             (FP64, for chi^2)
// The plain FP64 path (linalg.cu, psf.cu, ozaki.cu, cholfp64.cu) computes the same
// quantities at FP64 accuracy; the mixed path's deviation from it is measured by the tests.
#include <cuda.h>
#include <cuda_fp16.h>
#include <climits>
#include <cstring>
#include <algorithm>
#include "qlpix_ctx.h"
#include "chol.cuh"
#include "tc_syrk.cuh"
#include "tma_map.h"
#include "psf_tiles.cuh"
#include "chol128.cuh"

namespace qlpix {

#define MIXED_SOLVES 5    // solves of one evaluation: one and up to four refinement sweeps

struct MixedWork {
    void* base = nullptr;    // the allocation that holds all but F0
    double* t = nullptr;     // N (image-plane scratch)
    Csc csc{};               // L by source cell, for k_psf_x and L^T
    float* F0 = nullptr;     // lambda optimisation: X X^T before lambda R (allocated on first use)
    __half* X_hi = nullptr;  // F16 parts of X
    __half* X_lo = nullptr;
    int K_cap = 0;           // columns of X (image pixels), multiple of 32
    int M_cap = 0;           // rows of X, multiple of 128
    unsigned char* nz = nullptr;
    int nkb_cap = 0;
    float* F32 = nullptr;
    float* R32 = nullptr;
    int ld32 = 0;
    double* u = nullptr;     // N
    double* v = nullptr;     // M
    double* r = nullptr;     // M
    double* z = nullptr;     // M
    double* y = nullptr;     // M (solve scratch)
    double* img = nullptr;   // npix_pad: dense padded image for the FP64 convolutions
    float* linvF = nullptr;  // per 128-block of F: inverse of its diagonal factor, then its transpose
    float* yf = nullptr;     // M_cap: forward-solve result
    float* zf = nullptr;     // M_cap: backward-solve result (FP32 copy read by other CTAs)
    int* flags = nullptr;    // per solve 2 x nb: per-block "published" flags of the two sweeps
    int nb = 0;              // 128-blocks of M_cap
    CUtensorMap map_hi, map_lo;
    // the factorisations of F and R (k_chol128; concurrent, R on the side stream)
    Flow128Mem cf{}, cr{};
    CUtensorMap cf_maps[4], cr_maps[4];   // the split factor hi, lo and the split inverses hi, lo
    bool ready = false;
};

static MixedWork* mw_of(Slot& s) { return reinterpret_cast<MixedWork*>(s.mixed); }

// 128-row boxes of 128 bytes (64 F16 or 32 FP32 values), 128-byte swizzle
static int make_map(CUtensorMap* map, void* base, int rows, int cols, bool half)
{
    return make_map_box(map, base, rows, cols, half, TC_TILE, half ? 64 : 32);
}

// ---------------------------------------------------------------------------
// X = (P L sqrt(C^-1))^T as F16 hi + lo, and the nonzero flags of its
// 128-cell x 32-pixel blocks.
//
// Row s of X is the PSF-convolved image of source cell s: every pixel q that
// sees s (column s of the pre-PSF L) contributes L[q][s] to its PSF neighbours
// p with weight psf[k][l] (the transpose of QLens's gather,
// pixelgrid.cpp:14126-14168); the sum at p is then scaled by sqrt(C^-1) of p.
// The sums are 64-bit fixed point, so they are exact and independent of the
// order of the entries: each product is the exact product of two 32-bit
// integers, the tap on its grid (StaticData::psf_int) and the L entry on the
// grid 2^-PSFX_LEXP (2^-28: 4e-9 absolute, far below FP32 resolution of the
// entries) -- one wide multiply per tap.  No dense L' is stored.
// ---------------------------------------------------------------------------

// One entry of X split into F16 hi + lo parts of v scaled by xs (a power of two that
// puts X's largest entry near 2^14, undone exactly by the SYRK).  Returns whether
// either part is nonzero.
__device__ __forceinline__ bool store_x(__half* Xh, __half* Xl, size_t idx, float v, float xs)
{
    const float vs = v * xs;
    const __half h = __float2half_rn(vs);
    const __half l = __float2half_rn(vs - __half2float(h));
    Xh[idx] = h;
    Xl[idx] = l;
    return __half2float(h) != 0.0f || __half2float(l) != 0.0f;
}

// column counts of the merged pre-PSF L, the image tiles with active pixels, and the
// image pixel -> (active row, sqrt(C^-1)) table that k_psf_x reads: x fastest,
// with a border of half a PSF on every side so that no tap needs a bounds
// check (pixT[(j + pny/2) * (nx + 2 (pnx/2)) + i + pnx/2]; the rows of
// inactive and border pixels stay -1)
__global__ void k_csc_count(StaticData sd, const GridState* __restrict__ gs, const int* __restrict__ rowptr,
                            const int* __restrict__ cidx, const int* __restrict__ ccnt,
                            const double* __restrict__ cvec, const int* __restrict__ rowpix,
                            int* __restrict__ colcnt, int2* __restrict__ pixT, int ntx,
                            unsigned* __restrict__ active)
{
    const int N = gs->N;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x) {
        const int b = rowptr[r], n = ccnt[r];
        for (int e = 0; e < n; e++) atomicAdd(&colcnt[cidx[b + e]], 1);
        const float sq = sqrtf((float)cvec[r]);
        const int pix = rowpix[r];
        const int i = pix / sd.ny, j = pix - i * sd.ny;
        const int nxp = sd.nx + 2 * (sd.pnx / 2);
        pixT[(size_t)(j + sd.pny / 2) * nxp + i + sd.pnx / 2] = make_int2(r, __float_as_int(sq));
        const int tile = j / PSFX_R * ntx + i / 32;
        if (!(active[tile >> 5] >> (tile & 31) & 1u)) atomicOr(&active[tile >> 5], 1u << (tile & 31));
    }
}

// exclusive scan of colcnt[0..M) in place (colcnt[M] = total), cursor = starts
__global__ void __launch_bounds__(1024) k_csc_scan(const GridState* __restrict__ gs, int* __restrict__ colcnt,
                                                   int* __restrict__ cursor)
{
    __shared__ int part[1024];
    const int M = gs->M;
    const int per = (M + 1023) / 1024;
    const int a = threadIdx.x * per, b = min(a + per, M);
    int sum = 0;
    for (int i = a; i < b; i++) sum += colcnt[i];
    part[threadIdx.x] = sum;
    __syncthreads();
    for (int off = 1; off < 1024; off <<= 1) {     // Hillis-Steele inclusive scan
        int v = (threadIdx.x >= off) ? part[threadIdx.x - off] : 0;
        __syncthreads();
        part[threadIdx.x] += v;
        __syncthreads();
    }
    int run = part[threadIdx.x] - sum;
    for (int i = a; i < b; i++) {
        const int c = colcnt[i];
        colcnt[i] = run;
        cursor[i] = run;
        run += c;
    }
    if (threadIdx.x == 1023) colcnt[M] = part[1023];
}

__global__ void k_csc_fill(const GridState* __restrict__ gs, const int* __restrict__ rowptr,
                           const int* __restrict__ cidx, const int* __restrict__ ccnt, int* __restrict__ cursor,
                           int* __restrict__ col_u, int* __restrict__ src_u)
{
    const int N = gs->N;
    for (int r = blockIdx.x * blockDim.x + threadIdx.x; r < N; r += gridDim.x * blockDim.x) {
        const int b = rowptr[r], n = ccnt[r];
        for (int e = 0; e < n; e++) {
            const int pos = atomicAdd(&cursor[cidx[b + e]], 1);
            col_u[pos] = r;
            src_u[pos] = b + e;
        }
    }
}

// Entry k of the sorted columns: as the PSF-to-X build reads it (its pixel and L
// on its grid) with its row and FP64 value, or (fine) as the plain path's build
// of L' does, on the cell's grid (shift).
__device__ __forceinline__ void csc_store(const Csc& o, int k, int row, double v, const int* __restrict__ rowpix, int ny,
                                          int shift)
{
    const int pix = rowpix[row], i = pix / ny, j = pix - i * ny;
    if (o.fine) {
        o.fine[k] = o.raw ? psf64_raw(i, j, v) : psf64_entry(i, j, v, shift);
        return;
    }
    o.colrow[k] = row;
    o.ent[k] = make_int2((i << 16) | j, __float2int_rn((float)v * ldexpf(1.0f, PSFX_LEXP)));
    o.colval64[k] = v;
}

// Each column's entries in increasing row order, so that every sum over a
// column runs in a fixed order (k_csc_fill places them in atomic order).
// Rows are distinct within a column of the merged L, so the order is a
// permutation: columns of up to CSC_SORT_WARP entries are sorted by a warp in
// registers (k_csc_sort_w), longer ones by a CTA that marks their rows in a bitmap
// and takes each entry's rank from the marks below it.
#define CSC_SORT_WARP 64    // columns sorted a warp each (k_csc_sort_w)
#define CSC_WORDS 4096      // bitmap words a pass: 131,072 rows
// Columns of up to CSC_SORT_WARP entries, a warp each: the same permutation
// by a bitonic network in registers (R = 1 or 2 entries a lane, entry
// lane + 32 h in register h; partners 32 apart within the lane, the others
// through lane shuffles; no barriers); k_csc_sort takes the longer columns.
// The rows are distinct, so any sort gives the same order.
__device__ __forceinline__ void csc_bitonic_step(int& key, int& pos, int e, int j, int k)
{
    const int kp = __shfl_xor_sync(0xffffffffu, key, j), pp = __shfl_xor_sync(0xffffffffu, pos, j);
    const bool up = ((e & ~j) & k) == 0;                  // the pair's direction, from its lower index
    const bool take_min = ((e & j) == 0) == up;
    if (take_min ? (kp < key) : (kp > key)) { key = kp; pos = pp; }
}

template <int R>
__device__ __forceinline__ void csc_sort_warp(const int* __restrict__ col_u, const int* __restrict__ src_u,
                                              const double* __restrict__ cval, int b, int n, int lane,
                                              const Csc& out, const int* __restrict__ rowpix, int ny, int s)
{
    int key[R], pos[R];
    #pragma unroll
    for (int h = 0; h < R; h++) {
        const int e = lane + 32 * h;
        key[h] = (e < n) ? col_u[b + e] : INT_MAX;
        pos[h] = (e < n) ? src_u[b + e] : 0;
    }
    int shift = 0;
    if (out.fine) {
        int top = 0;
        #pragma unroll
        for (int h = 0; h < R; h++)
            if (lane + 32 * h < n) top = max(top, psf64_top(cval[pos[h]]));
        shift = psf64_shift(__reduce_max_sync(0xffffffffu, top));
        if (lane == 0) out.shift[s] = shift;
    }
    #pragma unroll
    for (int k = 2; k <= 32 * R; k <<= 1) {
        #pragma unroll
        for (int j = k >> 1; j > 0; j >>= 1) {
            if (j >= 32) {
                #pragma unroll
                for (int h = 0; h < R; h++) {
                    const int h2 = h ^ (j >> 5);
                    if (h2 > h) {
                        const bool up = ((lane + 32 * h) & k) == 0;
                        if ((key[h] > key[h2]) == up) {
                            const int tk = key[h]; key[h] = key[h2]; key[h2] = tk;
                            const int tp = pos[h]; pos[h] = pos[h2]; pos[h2] = tp;
                        }
                    }
                }
            } else {
                #pragma unroll
                for (int h = 0; h < R; h++) csc_bitonic_step(key[h], pos[h], lane + 32 * h, j, k);
            }
        }
    }
    #pragma unroll
    for (int h = 0; h < R; h++) {
        const int e = lane + 32 * h;
        if (e < n) csc_store(out, b + e, key[h], cval[pos[h]], rowpix, ny, shift);
    }
}

// Five barriers a pass, where a bitonic network took 28 to 45 (us, 3,700 columns of 60 to
// 300 entries 69 -> 11; 2,304 columns 37 -> 10).
__global__ void __launch_bounds__(256) k_csc_sort(const GridState* __restrict__ gs, const int* __restrict__ colptr,
                                                  const int* __restrict__ col_u, const int* __restrict__ src_u,
                                                  const double* __restrict__ cval, Csc out,
                                                  const int* __restrict__ rowpix, int ny, double* __restrict__ clear,
                                                  int ld)
{
    __shared__ unsigned bits[CSC_WORDS];
    __shared__ int below[CSC_WORDS];
    __shared__ int wsum[8];
    __shared__ int top;
    const int s = blockIdx.x;
    if (s >= gs->M) return;
    const int N = gs->N, b = colptr[s], n = colptr[s + 1] - b;
    if (clear) {
        double2* row = reinterpret_cast<double2*>(clear + (size_t)s * ld);
        for (int i = threadIdx.x; i < (N + 1) / 2; i += blockDim.x) row[i] = make_double2(0.0, 0.0);
    }
    if (n <= CSC_SORT_WARP) {
        if (clear && threadIdx.x < 32) {
            if (n <= 32) csc_sort_warp<1>(col_u, src_u, cval, b, n, threadIdx.x, out, rowpix, ny, s);
            else csc_sort_warp<2>(col_u, src_u, cval, b, n, threadIdx.x, out, rowpix, ny, s);
        }
        return;                                           // else k_csc_sort_w's
    }
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    int shift = 0;
    if (out.fine) {
        if (threadIdx.x == 0) top = 0;
        __syncthreads();
        int t = 0;
        for (int i = threadIdx.x; i < n; i += 256) t = max(t, psf64_top(cval[src_u[b + i]]));
        t = __reduce_max_sync(0xffffffffu, t);
        if (lane == 0) atomicMax(&top, t);
        __syncthreads();
        shift = psf64_shift(top);
        if (threadIdx.x == 0) out.shift[s] = shift;
    }
    int placed = 0;                                       // entries of the passes before
    for (int r0 = 0; r0 < N; r0 += 32 * CSC_WORDS) {
        const int words = min(CSC_WORDS, (N - r0 + 31) / 32);
        for (int w = threadIdx.x; w < words; w += 256) bits[w] = 0;
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += 256) {
            const unsigned r = (unsigned)(col_u[b + i] - r0);
            if (r < 32u * words) atomicOr(&bits[r >> 5], 1u << (r & 31));
        }
        __syncthreads();
        // the marks below each word: a thread a run of words, then a scan of the runs
        const int per = (words + 255) / 256, w0 = threadIdx.x * per, w1 = min(w0 + per, words);
        int sum = 0;
        for (int w = w0; w < w1; w++) sum += __popc(bits[w]);
        int at = sum;
        #pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const int v = __shfl_up_sync(0xffffffffu, at, o);
            if (lane >= o) at += v;
        }
        if (lane == 31) wsum[warp] = at;
        __syncthreads();
        int total = 0;
        #pragma unroll
        for (int w = 0; w < 8; w++) {
            if (w < warp) at += wsum[w];
            total += wsum[w];
        }
        at += placed - sum;
        for (int w = w0; w < w1; w++) {
            below[w] = at;
            at += __popc(bits[w]);
        }
        __syncthreads();
        for (int i = threadIdx.x; i < n; i += 256) {
            const int row = col_u[b + i];
            const unsigned r = (unsigned)(row - r0);
            if (r < 32u * words)
                csc_store(out, b + below[r >> 5] + __popc(bits[r >> 5] & ((1u << (r & 31)) - 1)), row,
                          cval[src_u[b + i]], rowpix, ny, shift);
        }
        placed += total;
        __syncthreads();
    }
}

__global__ void __launch_bounds__(256, 4) k_csc_sort_w(const GridState* __restrict__ gs,
                                                       const int* __restrict__ colptr,
                                                       const int* __restrict__ col_u, const int* __restrict__ src_u,
                                                       const double* __restrict__ cval, Csc out,
                                                       const int* __restrict__ rowpix, int ny)
{
    const int lane = threadIdx.x & 31;
    const int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (s >= gs->M) return;                                // whole warps
    const int b = colptr[s], n = colptr[s + 1] - b;
    if (n <= 32) csc_sort_warp<1>(col_u, src_u, cval, b, n, lane, out, rowpix, ny, s);
    else if (n <= CSC_SORT_WARP) csc_sort_warp<2>(col_u, src_u, cval, b, n, lane, out, rowpix, ny, s);
}

// out[s] = sum over column s of L of value * w[row]: one warp per column, lane
// l takes entries l, l+32, ... in row order, then a fixed shuffle tree; zero
// from M up to the 64-padding.
__global__ void __launch_bounds__(256) k_LTw_csc(const GridState* __restrict__ gs, const int* __restrict__ colptr,
                                                 const int* __restrict__ colrow,
                                                 const double* __restrict__ colval64, const double* __restrict__ w,
                                                 double* __restrict__ out)
{
    const int M = gs->M, Mp = (M + 63) & ~63;
    const int lane = threadIdx.x & 31;
    for (int s = blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); s < Mp; s += gridDim.x * (blockDim.x >> 5)) {
        double acc = 0;
        if (s < M) {
            const int b = colptr[s], e = colptr[s + 1];
            for (int k = b + lane; k < e; k += 32) acc += colval64[k] * w[colrow[k]];
        }
        for (int o = 16; o > 0; o >>= 1) acc += __shfl_xor_sync(0xffffffffu, acc, o);
        if (lane == 0) out[s] = acc;
    }
}

// int64 -> float, rounded to nearest even, in integer arithmetic (the same
// result as the conversion instruction, which GB300 issues to its FP64 pipe):
// the top 24 significant bits, rounded on the bits below them.
__device__ __forceinline__ float ll2f_rn_int(long long v)
{
    if (v == 0) return 0.0f;
    const unsigned sign = v < 0 ? 0x80000000u : 0u;
    const unsigned long long a = v < 0 ? 0ull - (unsigned long long)v : (unsigned long long)v;
    int e = 63 - __clzll((long long)a);          // index of the top bit
    unsigned m;
    if (e <= 23) {
        m = (unsigned)(a << (23 - e));
    } else {
        const int sh = e - 23;
        m = (unsigned)(a >> sh);
        const unsigned long long rem = a & ((1ull << sh) - 1), half = 1ull << (sh - 1);
        if (rem > half || (rem == half && (m & 1u))) {
            if (++m == (1u << 24)) { m >>= 1; e++; }
        }
    }
    return __uint_as_float(sign | ((unsigned)(e + 127) << 23) | (m & 0x7fffffu));
}

// X by image tiles of 32 pixels along x and PSFX_R rows.  k_psfx_tiles lists the
// tiles with active pixels that some footprint of a cell reaches, a warp a cell;
// k_psf_x gives each listed tile to a warp, lane x keeping its column's sums in
// registers and adding tap x L for every entry whose footprint meets the tile
// (found by the entries' sorted rows and a ballot over their columns; the taps
// carry a border of zeros, so that none is tested).  Every entry of X outside the
// listed tiles is zero: X is all zero between evaluations, k_x_clean takes the
// tiles back.
// Scattering a footprint tap by tap into shared memory took a 64-bit shared atomic
// a tap, which bounded it.  Now a tap is a 32-bit load from shared memory, which
// bounds it, and a wide multiply-add, 2 to 3 of them a useful one (tiles that a
// footprint fills in part; 16 rows were 10-40 % slower).  A warp's tiles come from
// all cells: with a CTA a cell, cells of many entries were left over at the end.
// us, before -> now: a 21 x 21 PSF and 3,500 cells on 11,800 pixels 263 -> 68, on
// 36,000 pixels 970 -> 118; a 31 x 31 PSF on 42,000 pixels 383 -> 180.
// PAD = false (PSFs whose bordered taps pass PSFX_PAD_BYTES): taps by their
// bounds from global memory.
template <bool PAD>
__global__ void __launch_bounds__(512) k_psf_x(StaticData sd, const int* __restrict__ colptr,
                                               const int2* __restrict__ ent_g, const int2* __restrict__ pixT, int ntx,
                                               const int* __restrict__ count, const uint2* __restrict__ list,
                                               __half* __restrict__ Xh, __half* __restrict__ Xl, float xs, int K_cap,
                                               unsigned char* __restrict__ nz, int nkb_cap)
{
    extern __shared__ __align__(16) int taps[];  // [pnx + 62][pitch]: column pk + 31, row pl + R - 1
    constexpr int R = PSFX_R;
    const int pnx = sd.pnx, pny = sd.pny, nxh = pnx / 2, nyh = pny / 2, nxp = sd.nx + 2 * nxh;
    const int pitch = psfx_pitch(pny);
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, items = *count;
    if ((int)blockIdx.x * nw >= items) return;
    if (PAD) {
        for (int t = threadIdx.x; t < (pnx + 62) * pitch; t += blockDim.x) {
            const int pk = t / pitch - 31, pl = t % pitch - (R - 1);
            taps[t] = (pk >= 0 && pk < pnx && pl >= 0 && pl < pny) ? sd.psf_int[pl * pnx + pk] : 0;
        }
        __syncthreads();
    }
    const float inv = ldexpf(1.0f, -sd.fix_exp_x);
    for (int it = blockIdx.x * nw + (threadIdx.x >> 5); it < items; it += gridDim.x * nw) {
        const uint2 item = list[it];
        const int s = item.x, y0 = (int)item.y / ntx * R, x0 = ((int)item.y % ntx) * 32, x = x0 + lane;
        const int n = colptr[s + 1] - colptr[s];
        const int2* ent = ent_g + colptr[s];
        int lo = 0, hi = n;
        if (n > 64) {
            lo = warp_lower_bound_row(ent, n, y0 + nyh - pny + 1);
            hi = warp_lower_bound_row(ent, n, y0 + R + nyh);
        }
        long long acc[R];
        #pragma unroll
        for (int r = 0; r < R; r++) acc[r] = 0;
        for (int e0 = lo; e0 < hi; e0 += 32) {
            int dx = -32, dy = 0, v = 0;
            if (e0 + lane < hi) {
                const int2 en = ent[e0 + lane];
                dx = x0 - ((en.x >> 16) - nxh);          // column of lane 0's tap
                dy = y0 - ((en.x & 0xffff) - nyh);       // row of the first row's tap
                v = en.y;
            }
            unsigned hit = __ballot_sync(0xffffffffu, dx > -32 && dx < pnx && dy > -R && dy < pny);
            for (; hit; hit &= hit - 1) {
                const int f = __ffs(hit) - 1;
                const int ox = __shfl_sync(0xffffffffu, dx, f) + lane, oy = __shfl_sync(0xffffffffu, dy, f);
                const long long ve = __shfl_sync(0xffffffffu, v, f);
                if (PAD) {
                    const int* tp = taps + (ox + 31) * pitch + oy + R - 1;
                    #pragma unroll
                    for (int r = 0; r < R; r++) acc[r] += (long long)tp[r] * ve;
                } else if (ox >= 0 && ox < pnx) {
                    #pragma unroll
                    for (int r = 0; r < R; r++)
                        if (oy + r >= 0 && oy + r < pny) acc[r] += (long long)sd.psf_int[(oy + r) * pnx + ox] * ve;
                }
            }
        }
        // X[s][row] for the tile's active pixels: sqrt(C^-1) times the sum, split into hi + lo
        if (x >= sd.nx) continue;
        #pragma unroll
        for (int r = 0; r < R; r++) {
            if (y0 + r >= sd.ny) break;
            const int2 pt = pixT[(size_t)(y0 + r + nyh) * nxp + x + nxh];
            if (pt.x < 0 || acc[r] == 0) continue;
            const float v = (ll2f_rn_int(acc[r]) * inv) * __int_as_float(pt.y);
            if (store_x(Xh, Xl, (size_t)s * K_cap + pt.x, v, xs))
                nz[(size_t)(s / TC_TILE) * nkb_cap + pt.x / TC_KB] = 1;
        }
    }
}

// After the SYRK has read X: the listed tiles' pixels back to zero (clearing all of
// X moved ~480 MB at 4,096 cells x 58,000 pixels).
__global__ void __launch_bounds__(256) k_x_clean(StaticData sd, const int2* __restrict__ pixT, int ntx,
                                                 const int* __restrict__ count, const uint2* __restrict__ list,
                                                 __half* __restrict__ Xh, __half* __restrict__ Xl, int K_cap)
{
    const int lane = threadIdx.x & 31, items = *count;
    const int nxh = sd.pnx / 2, nyh = sd.pny / 2, nxp = sd.nx + 2 * nxh;
    for (int it = blockIdx.x * 8 + (threadIdx.x >> 5); it < items; it += gridDim.x * 8) {
        const uint2 item = list[it];
        const int y0 = (int)item.y / ntx * PSFX_R, x = ((int)item.y % ntx) * 32 + lane;
        if (x >= sd.nx) continue;
        int row[PSFX_R];
        #pragma unroll
        for (int r = 0; r < PSFX_R; r++)
            row[r] = y0 + r < sd.ny ? pixT[(size_t)(y0 + r + nyh) * nxp + x + nxh].x : -1;
        #pragma unroll
        for (int r = 0; r < PSFX_R; r++) {
            if (row[r] < 0) continue;
            const size_t idx = (size_t)item.x * K_cap + row[r];
            Xh[idx] = __float2half_rn(0.0f);
            Xl[idx] = __float2half_rn(0.0f);
        }
    }
}

// F32 += lambda R; R32 = R; identity beyond M up to the 64-padding.
__device__ __forceinline__ int act_at32(const int* ai, int snx, int sny, int i, int j)
{
    if (i < 0 || j < 0 || i >= snx || j >= sny) return -1;
    return ai[j * snx + i];
}

__global__ void k_reg32(const GridState* __restrict__ gs, const int* __restrict__ ai,
                        const double* __restrict__ regp, float* __restrict__ F, float* __restrict__ R, int ld,
                        int do_reg, int parts)
{
    const bool toF = parts & REG_F, toR = parts & REG_R;
    const double regparam = *regp;
    const int snx = gs->snx, sny = gs->sny;
    const int M = gs->M, Mp = (M + 127) & ~127;   // identity up to the 128-block padding
    const int ncell = snx * sny;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell + (Mp - M); c += gridDim.x * blockDim.x) {
        if (c >= ncell) {
            int i = M + (c - ncell);
            if (toF) F[(size_t)i * ld + i] = 1.0f;
            if (do_reg && toR) R[(size_t)i * ld + i] = 1.0f;
            continue;
        }
        if (!do_reg) continue;
        const int a = ai[c];
        if (a < 0) continue;
        const int ci = c % snx, cj = c / snx;
        int nb1[4] = {act_at32(ai, snx, sny, ci + 1, cj), act_at32(ai, snx, sny, ci - 1, cj),
                      act_at32(ai, snx, sny, ci, cj + 1), act_at32(ai, snx, sny, ci, cj - 1)};
        int nb2[4] = {act_at32(ai, snx, sny, ci + 2, cj), act_at32(ai, snx, sny, ci - 2, cj),
                      act_at32(ai, snx, sny, ci, cj + 2), act_at32(ai, snx, sny, ci, cj - 2)};
        double diag = 8.0;
        for (int k = 0; k < 4; k++) if (nb1[k] >= 0) diag += 1.0;
        if (toR) R[(size_t)a * ld + a] = (float)diag;
        if (toF) F[(size_t)a * ld + a] = (float)((double)F[(size_t)a * ld + a] + regparam * diag);
        for (int k = 0; k < 4; k++) {
            int b = nb1[k];
            if (b >= 0 && b < a) {
                if (toR) R[(size_t)a * ld + b] = -4.0f;
                if (toF) F[(size_t)a * ld + b] = (float)((double)F[(size_t)a * ld + b] - 4.0 * regparam);
            }
            int b2 = nb2[k];
            if (b2 >= 0 && nb1[k] >= 0 && b2 < a) {
                if (toR) R[(size_t)a * ld + b2] = 1.0f;
                if (toF) F[(size_t)a * ld + b2] = (float)((double)F[(size_t)a * ld + b2] + regparam);
            }
        }
    }
}

// ---------------------------------------------------------------------------
// FP64 refinement pieces
// ---------------------------------------------------------------------------
__global__ void k_copy_init(const GridState* __restrict__ gs, const double* __restrict__ D, double* __restrict__ r,
                            double* __restrict__ s)
{
    const int Mp = (gs->M + 63) & ~63;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < Mp; i += gridDim.x * blockDim.x) {
        r[i] = D[i];
        s[i] = 0.0;
    }
}

__global__ void k_axpy(const GridState* __restrict__ gs, const double* __restrict__ z, double* __restrict__ s)
{
    const int Mp = (gs->M + 63) & ~63;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < Mp; i += gridDim.x * blockDim.x) s[i] += z[i];
}

// r = D - v - lambda R s   (v = L'^T C^-1 L' s; R applied by its stencil)
__global__ void k_residual(const GridState* __restrict__ gs, const double* __restrict__ D,
                           const double* __restrict__ vv, const int* __restrict__ ai,
                           const double* __restrict__ regp, int do_reg, const double* __restrict__ s,
                           double* __restrict__ r)
{
    const double regparam = *regp;
    const int snx = gs->snx, sny = gs->sny;
    const int M = gs->M;
    const int ncell = snx * sny;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell; c += gridDim.x * blockDim.x) {
        const int a = ai[c];
        if (a < 0) continue;
        const double v = vv[a];
        double rs = 0;
        if (do_reg) {
            const int ci = c % snx, cj = c / snx;
            int nb1[4] = {act_at32(ai, snx, sny, ci + 1, cj), act_at32(ai, snx, sny, ci - 1, cj),
                          act_at32(ai, snx, sny, ci, cj + 1), act_at32(ai, snx, sny, ci, cj - 1)};
            int nb2[4] = {act_at32(ai, snx, sny, ci + 2, cj), act_at32(ai, snx, sny, ci - 2, cj),
                          act_at32(ai, snx, sny, ci, cj + 2), act_at32(ai, snx, sny, ci, cj - 2)};
            double diag = 8.0;
            for (int k = 0; k < 4; k++) {
                if (nb1[k] >= 0) { diag += 1.0; rs += -4.0 * s[nb1[k]]; }
                if (nb2[k] >= 0 && nb1[k] >= 0) rs += s[nb2[k]];
            }
            rs += diag * s[a];
        }
        r[a] = D[a] - v - regparam * rs;
    }
    (void)M;
}

// ---------------------------------------------------------------------------
void mixed_free(Slot& c)
{
    MixedWork* m = mw_of(c);
    if (!m) return;
    void* ptrs[] = {m->base, m->F0};
    for (void* p : ptrs) if (p) cudaFree(p);
    delete m;
    c.mixed = nullptr;
}

void csc_free(Csc& o)
{
    if (o.base) cudaFree(o.base);
    o = Csc{};
}

// L by source cell for M_cap cells of a slot; fine: the plain path's.
void csc_layout(Csc& o, const Slot& c, int M_cap, bool fine, Arena& ar)
{
    const int ntile = (c.img_nx + 31) / 32 * ((c.img_ny + PSFX_R - 1) / PSFX_R);
    const size_t nnz = (size_t)3 * c.N_cap * c.nsub_cap;
    o.words = (ntile + 31) / 32;
    o.M_cap = M_cap;
    o.npix_pad = c.npix_pad;
    ar.add(&o.tiles, (size_t)M_cap * std::min(ntile, c.N_cap));
    ar.add(&o.tile_active, o.words + 1);
    ar.add(&o.colcnt, M_cap + 1);
    ar.add(&o.cursor, M_cap);
    ar.add(&o.col_u, nnz);
    ar.add(&o.src_u, nnz);
    ar.add(&o.pixT, c.npix_pad);
    if (fine) {
        ar.add(&o.fine, nnz);
        ar.add(&o.shift, M_cap);
    } else {
        ar.add(&o.colrow, nnz);
        ar.add(&o.ent, nnz);
        ar.add(&o.colval64, nnz);
    }
}

void csc_clear(const Csc& o, ClearList& l)
{
    l.add(o.colcnt, sizeof(int) * (size_t)(o.M_cap + 1));
    l.add(o.tile_active, sizeof(unsigned) * (o.words + 1));
    l.add(o.pixT, sizeof(int2) * (size_t)o.npix_pad, 0xffffffffu);
}

// L by source cell (CSC, rows ascending within a column) and the list of the
// (cell, tile) pairs that its footprints reach.  clear: M rows of N of the plain
// path's L', set to zero on the way.
void launch_csc(const StaticData& sd, const Work& w, const Csc& o, int N_cap, double* clear, int ld, cudaStream_t st)
{
    const int rb = std::max(1, std::min((N_cap + 255) / 256, 152 * 8)), ntx = (sd.nx + 31) / 32;
    k_csc_count<<<rb, 256, 0, st>>>(sd, w.gs, w.rowptr, w.cidx, w.ccnt, w.cvec, w.rowpix, o.colcnt, o.pixT, ntx,
                                    o.tile_active);
    k_csc_scan<<<1, 1024, 0, st>>>(w.gs, o.colcnt, o.cursor);
    k_csc_fill<<<rb, 256, 0, st>>>(w.gs, w.rowptr, w.cidx, w.ccnt, o.cursor, o.col_u, o.src_u);
    // the plain path's CTAs are there for the clearing anyway and take the short columns too
    if (!clear)
        k_csc_sort_w<<<(o.M_cap + 7) / 8, 256, 0, st>>>(w.gs, o.colcnt, o.col_u, o.src_u, w.cval, o, w.rowpix, sd.ny);
    k_csc_sort<<<o.M_cap, 256, 0, st>>>(w.gs, o.colcnt, o.col_u, o.src_u, w.cval, o, w.rowpix, sd.ny, clear, ld);
    const int span = std::min(o.words, 48 * 1024 / (int)sizeof(unsigned));
    const size_t wmark = sizeof(unsigned) * span;
    const int tw = (int)std::max<size_t>(1, std::min<size_t>(8, 48 * 1024 / wmark));      // cells a CTA
    if (o.fine)
        k_psfx_tiles<<<(o.M_cap + tw - 1) / tw, 32 * tw, wmark * tw, st>>>(sd, w.gs, o.colcnt, o.fine, ntx, o.words, span,
                                                                          o.tile_active, o.ntiles(), o.tiles);
    else
        k_psfx_tiles<<<(o.M_cap + tw - 1) / tw, 32 * tw, wmark * tw, st>>>(sd, w.gs, o.colcnt, o.ent, ntx, o.words, span,
                                                                          o.tile_active, o.ntiles(), o.tiles);
    count_launches(clear ? 5 : 6);
}

// R couples a cell to cells at most two grid rows (2 snx active indices) away.
static int band128_R(int snx) { return (2 * snx - 1) / C2 + 1; }

static size_t flow128_flags(int nb) { return (size_t)nb * nb + nb + 1; }

static int flow_maps(const Flow128Mem& f, CUtensorMap* maps)
{
    for (int k = 0; k < 2; k++) {
        int r = make_map(&maps[k], k ? f.Ll : f.Lh, f.rows, f.wb * C2, true);
        if (r == QLP_OK) r = make_map(&maps[2 + k], k ? f.il : f.ih, f.rows, C2, false);
        if (r != QLP_OK) return r;
    }
    return QLP_OK;
}

int mixed_init(Slot& c)
{
    MixedWork* m = mw_of(c);
    const int M_cap = (c.M_cap + TC_TILE - 1) / TC_TILE * TC_TILE;
    const int K_cap = (c.N_cap + TC_KB - 1) / TC_KB * TC_KB + TC_KB;
    if (m && m->ready && m->M_cap >= M_cap && m->K_cap >= K_cap) return QLP_OK;
    mixed_free(c);
    m = new MixedWork();
    c.mixed = m;
    m->M_cap = M_cap;
    m->K_cap = K_cap;
    m->nkb_cap = K_cap / TC_KB;
    m->ld32 = M_cap;
    Arena ar;
    auto A = [&](void** p, size_t bytes) { ar.add(reinterpret_cast<char**>(p), bytes); };
    const size_t xbytes = sizeof(__half) * (size_t)M_cap * K_cap;
    A((void**)&m->X_hi, xbytes);
    A((void**)&m->X_lo, xbytes);
    A((void**)&m->nz, (size_t)(M_cap / TC_TILE) * m->nkb_cap + 3);
    A((void**)&m->F32, sizeof(float) * (size_t)M_cap * M_cap);
    A((void**)&m->R32, sizeof(float) * (size_t)M_cap * M_cap);
    A((void**)&m->img, sizeof(double) * (size_t)c.npix_pad);
    csc_layout(m->csc, c, M_cap, false, ar);
    A((void**)&m->t, sizeof(double) * (size_t)(c.N_cap + 64));
    A((void**)&m->u, sizeof(double) * (size_t)(c.N_cap + 64));
    A((void**)&m->v, sizeof(double) * M_cap);
    A((void**)&m->r, sizeof(double) * M_cap);
    A((void**)&m->z, sizeof(double) * M_cap);
    A((void**)&m->y, sizeof(double) * M_cap);
    m->nb = M_cap / C2;
    A((void**)&m->linvF, sizeof(float) * (size_t)m->nb * 2 * C2 * C2);
    A((void**)&m->yf, sizeof(float) * (size_t)M_cap);
    A((void**)&m->zf, sizeof(float) * (size_t)M_cap);
    A((void**)&m->flags, sizeof(int) * (size_t)2 * m->nb * MIXED_SOLVES);
    for (Flow128Mem* f : {&m->cf, &m->cr}) {
        f->rows = M_cap;
        f->wb = f == &m->cr ? std::min(m->nb, band128_R(c.snx_cap) + 1) : m->nb;
        A((void**)&f->Lh, sizeof(__half) * (size_t)M_cap * f->wb * C2);
        A((void**)&f->Ll, sizeof(__half) * (size_t)M_cap * f->wb * C2);
        A((void**)&f->pexp, sizeof(int) * (size_t)m->nb * M_cap);
        A((void**)&f->ih, sizeof(float) * (size_t)M_cap * C2);
        A((void**)&f->il, sizeof(float) * (size_t)M_cap * C2);
        A((void**)&f->flags, sizeof(int) * flow128_flags(m->nb));
    }
    const cudaError_t e = ar.commit(&m->base);
    if (e != cudaSuccess) {
        set_error("%s (%d)", "mixed-precision workspace allocation failed", (int)e);
        return QLP_ERR_NOMEM;
    }
    cudaMemset(m->X_hi, 0, xbytes);
    cudaMemset(m->X_lo, 0, xbytes);
    cudaStreamSynchronize(0);                              // the slots' streams do not wait for stream 0
    if (make_map(&m->map_hi, m->X_hi, M_cap, K_cap, true) != QLP_OK ||
        make_map(&m->map_lo, m->X_lo, M_cap, K_cap, true) != QLP_OK ||
        flow_maps(m->cf, m->cf_maps) != QLP_OK || flow_maps(m->cr, m->cr_maps) != QLP_OK) {
        set_error("%s (%d)", "cuTensorMapEncodeTiled unavailable or failed", 0);
        return QLP_ERR_CUDA;
    }
    // shared-memory opt-ins (a kernel's static and dynamic shared memory
    // together may not pass 227 KB): a failed opt-in is reported here, not at
    // the first launch that needs it
    {
        cudaError_t ea = cudaSuccess;
        auto opt = [&](const void* f, int bytes) {
            const cudaError_t r = cudaFuncSetAttribute(f, cudaFuncAttributeMaxDynamicSharedMemorySize, bytes);
            if (ea == cudaSuccess) ea = r;
        };
        opt((const void*)k_psf_x<true>, 227 * 1024);
        opt((const void*)k_psf_x<false>, 227 * 1024);
        opt((const void*)k_chol128, C2_SMEM);
        opt((const void*)k_syrk_tc, TC_SMEM);
        if (ea != cudaSuccess) {
            set_error("%s (%d)", "shared-memory opt-in failed", (int)ea);
            return QLP_ERR_CUDA;
        }
    }
    m->ready = true;
    return QLP_OK;
}

// FP32 Cholesky of the mixed path (k_chol128).  band: 128-blocks below the
// diagonal that can be nonzero (the whole matrix for F); linv: per diagonal
// block its inverse and the inverse's transpose for the solves, or null; ctas:
// the grid's size.
static void cholesky_mixed(float* A, int ld, GridState* gs, int which, int band, float* linv, const Flow128Mem& f,
                           const CUtensorMap* maps, int ctas, cudaStream_t st)
{
    const int nb = f.rows / C2;
    const int tiles = nb * std::min(nb, band + 1);
    ctas = std::min(tiles, ctas);
    k_chol128<<<ctas, C2_THREADS, C2_SMEM, st>>>(maps[0], maps[1], maps[2], maps[3], A,
                                                                             ld, gs, which, band, f, linv);
}

// The lambda optimisation's F0 = X X^T (before lambda R): allocated outside
// any stream capture, before the first PIPE_PRE / PIPE_TRIAL sequence.
int mixed_ensure_f0(Slot& slot)
{
    int rc = mixed_init(slot);
    if (rc != QLP_OK) return rc;
    MixedWork* m = mw_of(slot);
    if (m->F0) return QLP_OK;
    if (cudaMalloc(&m->F0, sizeof(float) * (size_t)m->ld32 * m->M_cap) != cudaSuccess) {
        m->F0 = nullptr;
        set_error("%s (%d)", "lambda optimisation workspace allocation failed", m->M_cap);
        return QLP_ERR_NOMEM;
    }
    return QLP_OK;
}

const float* mixed_factor(Slot& slot, int& ld)
{
    ld = mw_of(slot)->ld32;
    return mw_of(slot)->F32;
}

// What an evaluation (or one lambda trial) starts from cleared.
void mixed_clear(Slot& slot, ClearList& l, bool trial)
{
    MixedWork* m = mw_of(slot);
    l.add(m->cf.flags, sizeof(int) * flow128_flags(m->nb));
    l.add(m->flags, sizeof(int) * (size_t)2 * m->nb * MIXED_SOLVES);
    if (trial) return;
    l.add(m->cr.flags, sizeof(int) * flow128_flags(m->nb));
    l.add(m->nz, (size_t)(m->M_cap / TC_TILE) * m->nkb_cap);
    csc_clear(m->csc, l);
    l.add(m->img, sizeof(double) * (size_t)slot.npix_pad);
}

// part: PIPE_ALL the whole inversion at the slot's lambda; PIPE_PRE everything
// that does not depend on lambda (D, X, F0 = X X^T kept aside, R and its log
// det); PIPE_TRIAL one lambda of the optimisation (F = F0 + lambda R, its
// factor, log det and the refined amplitudes, the model image).
int run_inversion_mixed(const qlp_ctx* c, Slot& slot, const StaticData& sd, const SrcOpts& so, const double* regp,
                        int part, cudaStream_t st, cudaEvent_t* ev)
{
    const int refine = c->refine;
    int rc = mixed_init(slot);
    if (rc != QLP_OK) return rc;
    MixedWork* m = mw_of(slot);
    Work& w = slot.w;
    const int N_cap = sd.n_mask;
    const int Mc = slot.M_cap;
    const int ltw_blocks = (m->M_cap + 7) / 8;
    int n = 0;
    if (part != PIPE_ALL && !m->F0) {
        set_error("%s (%d)", "lambda optimisation workspace missing", part);
        return QLP_ERR_ARG;
    }
    if (part == PIPE_TRIAL) {
        ClearList cl;
        cl.add(&w.gs->not_spd_F, sizeof(int));
        mixed_clear(slot, cl, true);
        rc = launch_clear(cl, st);
        if (rc != QLP_OK) return rc;
        launch_copy_square(m->F32, m->F0, m->ld32, 4, C2, w.gs, m->M_cap, st);
        k_reg32<<<(so.snx * so.sny + 128 + 255) / 256, 256, 0, st>>>(w.gs, w.active_index, regp, m->F32, m->R32,
                                                                    m->ld32, so.regularization, REG_F);
        n++;
    } else {

    if (so.regularization) {
        // R hangs on the active cells alone: its factorisation (log det R only)
        // runs on the slot's second stream beside everything up to the evidence,
        // within R's band.
        const int band_R = band128_R(so.snx);
        cudaEventRecord(slot.side_fork, st);
        cudaStreamWaitEvent(slot.side, slot.side_fork, 0);
        launch_clear_band(m->R32, m->ld32, 4, m->M_cap, C2, band_R, w.gs, slot.side);
        k_reg32<<<(so.snx * so.sny + 128 + 255) / 256, 256, 0, slot.side>>>(w.gs, w.active_index, regp, m->F32, m->R32,
                                                                           m->ld32, so.regularization, REG_R);
        cholesky_mixed(m->R32, m->ld32, w.gs, 1, band_R, nullptr, m->cr, m->cr_maps, 2, slot.side);
        k_logdet_t<float><<<1, 1024, 0, slot.side>>>(m->R32, m->ld32, w.gs, w.out);
        n += 3;
        cudaEventRecord(slot.side_join, slot.side);
    }
    launch_csc(sd, w, m->csc, N_cap, nullptr, 0, st);
    // D = L^T P^T (C^-1 d), FP64
    op_conv(sd, w, N_cap, true, w.dvec, w.cvec, m->t, m->img, m->csc.pixT, st);
    k_LTw_csc<<<ltw_blocks, 256, 0, st>>>(w.gs, m->csc.colcnt, m->csc.colrow, m->csc.colval64, m->t, w.D);
    n++;
    // X = (P L sqrt(C^-1))^T and its block flags, from L by source cell
    const float xs = ldexpf(1.0f, sd.x_exp);                      // F16 scale of X
    const int ntx = (sd.nx + 31) / 32;
    const int* ntiles = m->csc.ntiles();
    {
        const int pt = (c->psfx_threads == 128 || c->psfx_threads == 512) ? c->psfx_threads : 256;
        const size_t taps = sizeof(int) * psfx_taps(sd.pnx, sd.pny);
        const bool pad = taps <= PSFX_PAD_BYTES;
        auto k = pad ? k_psf_x<true> : k_psf_x<false>;
        k<<<152 * 1024 / pt, pt, pad ? taps : 0, st>>>(sd, m->csc.colcnt, m->csc.ent, m->csc.pixT, ntx, ntiles, m->csc.tiles, m->X_hi,
                                                       m->X_lo, xs, m->K_cap, m->nz, m->nkb_cap);
        n++;
    }
    if (ev) cudaEventRecord(ev[3], st);
    {
        const int nt = m->M_cap / TC_TILE;
        k_syrk_tc<<<nt * (nt + 1) / 2, 128, TC_SMEM, st>>>(m->map_hi, m->map_lo, w.gs, m->nz, m->nkb_cap, m->F32,
                                                           m->ld32, ldexpf(1.0f, -2 * sd.x_exp));
        n++;
        // X back to all zero for the next evaluation
        k_x_clean<<<152 * 8, 256, 0, st>>>(sd, m->csc.pixT, ntx, ntiles, m->csc.tiles, m->X_hi, m->X_lo, m->K_cap);
        n++;
    }
    if (ev) cudaEventRecord(ev[4], st);
    if (part == PIPE_PRE) launch_copy_square(m->F0, m->F32, m->ld32, 4, C2, w.gs, m->M_cap, st);
    if (part == PIPE_PRE) {
        if (so.regularization) cudaStreamWaitEvent(st, slot.side_join, 0);
        count_launches(n);
        return QLP_OK;
    }
    k_reg32<<<(so.snx * so.sny + 128 + 255) / 256, 256, 0, st>>>(w.gs, w.active_index, regp, m->F32, m->R32,
                                                                m->ld32, so.regularization, REG_F);
    n++;
    }   // part != PIPE_TRIAL
    cholesky_mixed(m->F32, m->ld32, w.gs, 0, 1 << 20, m->linvF, m->cf, m->cf_maps, factor_ctas(c, m->nb), st);
    n++;
    if (so.regularization && part == PIPE_ALL) cudaStreamWaitEvent(st, slot.side_join, 0);
    // s = F^-1 D with `refine` FP64 refinement sweeps
    k_copy_init<<<(Mc + 255) / 256, 256, 0, st>>>(w.gs, w.D, m->r, w.s);
    n++;
    for (int it = 0; it <= refine; it++) {
        int* const tf = m->flags + (size_t)it * 2 * m->nb;
        k_trsv128_fwd<<<m->nb, 256, 0, st>>>(m->F32, m->ld32, m->linvF, w.gs, m->r, m->yf, tf);
        k_trsv128_bwd<<<m->nb, 256, 0, st>>>(m->F32, m->ld32, m->linvF, w.gs, m->yf, m->zf, m->z,
                                              tf + m->nb);
        k_axpy<<<(Mc + 255) / 256, 256, 0, st>>>(w.gs, m->z, w.s);
        n += 3;
        if (it == refine) break;
        op_Ls(w, N_cap, w.s, m->t, st);
        op_conv(sd, w, N_cap, false, m->t, nullptr, m->u, m->img, m->csc.pixT, st);
        op_conv(sd, w, N_cap, true, m->u, w.cvec, m->t, m->img, m->csc.pixT, st);
        k_LTw_csc<<<ltw_blocks, 256, 0, st>>>(w.gs, m->csc.colcnt, m->csc.colrow, m->csc.colval64, m->t, m->v);
        n++;
        k_residual<<<(so.snx * so.sny + 255) / 256, 256, 0, st>>>(w.gs, w.D, m->v, w.active_index, regp,
                                                                  so.regularization, w.s, m->r);
        n++;
    }
    // model image P L s in FP64 for chi^2
    op_Ls(w, N_cap, w.s, m->t, st);
    op_conv(sd, w, N_cap, false, m->t, nullptr, w.model, m->img, m->csc.pixT, st);
    count_launches(n);
    return QLP_OK;
}

}  // namespace qlpix
