// psf.cu -- PSF convolution of the lensing matrix into the plain path's dense L',
// kept by source cell.
//
// QLens::PSF_convolution_Lmatrix_dense, direct path (pixelgrid.cpp:14092-14176):
//   L'[p][s] = sum over PSF taps (k-major, then l) of psf[k][l] * Ldense[q][s],
//   q = the active pixel at (i_p + nx/2 - k, j_p + ny/2 - l).
// The sums are exact in 64-bit fixed point (psf_tiles.cuh, StaticData::psf_fine):
// L to 2^-57 of the power of two below the cell's largest, the taps to 2^-51 or better of the largest (2^-57 for a
// Gaussian of 21 x 21), by halves; of a product (th 2^w + tl) (vh 2^29 + vl) only
// tl vl is left out, below 2^-59 of the largest tap where that is an eighth of their
// sum.  An FP64 sum rounds at 2^-53 of each product and partial sum.  Other PSFs, and
// noise maps that weight small entries up past those bounds, are summed in FP64
// (psf_fixed_rule, ctx.cpp).
#include "qlpix_ctx.h"
#include "psf_tiles.cuh"

namespace qlpix {

// outside the normal numbers; out of line, for eight of them inlined cost more to fetch
// than a small problem's sums
__device__ __noinline__ double fixed_scaled(long long s, int k) { return scalbn((double)s, -k); }

// s 2^-k, |s| < 2^63, rounded to nearest even; integer arithmetic (FP64 conversions
// go to the FP64 pipe) but for results outside the normal numbers.
__device__ __forceinline__ double fixed_to_double(long long s, int k)
{
    if (s == 0) return 0.0;
    unsigned long long a = s < 0 ? 0ull - (unsigned long long)s : (unsigned long long)s;
    int e = 63 - __clzll((long long)a);
    if (e + 1022 - k < 1 || e + 1024 - k > 2046) return fixed_scaled(s, k);
    if (e <= 52) {
        a <<= 52 - e;
    } else {
        const int sh = e - 52;
        const unsigned long long rem = a & ((1ull << sh) - 1), half = 1ull << (sh - 1);
        a >>= sh;
        if (rem > half || (rem == half && (a & 1))) a++;           // a carry to 2^53 moves the exponent below
    }
    const unsigned long long b = a + ((unsigned long long)(e + 1022 - k) << 52);
    return __longlong_as_double((long long)(b | (s < 0 ? 1ull << 63 : 0)));
}

// L' by image tiles, as k_psf_x builds X: a warp takes a listed (cell, 32 x 8
// pixels) pair, lane x keeps its column's sums and adds tap x L for every entry
// whose footprint meets the tile, three wide multiply-adds and a 64-bit load from
// shared memory a tap.  With the values go each cell's largest biased exponent (with a
// noise map of L' sqrt(C^-1), the digits' operand) and the live 32-pixel stages of each
// 64 cells, for the digits.
// At 24 warps an SM it waits on the chain from an entry to its taps and multiplies
// (shared memory 21 %, issue 36 % busy).  A warp per image row that scattered tapped
// rows into shared memory in FP64, a tap after the other, waited on those.  2,934 cells x
// 11,772 pixels, 441 taps: 1,940 -> 146 us (and 46 us for the entries by cell and
// the clearing of L'); 738 x 6,220, 49 taps: 101 -> 38 us; 16 uneven evaluations at
// up to 4,096 cells, 121 taps: 14.2 -> 10.4 ms.  In FP64 (below)
// the first takes 0.14 ms more.
// FIXED = false (StaticData::psf_fixed, or bordered taps past PSF64_PAD_BYTES): FP64
// sums of the FP64 entries, taps by their bounds from global memory.
#define PSF64_PAD_BYTES (200 * 1024)
template <bool FIXED>
__global__ void __launch_bounds__(256) k_psf64(StaticData sd, const GridState* __restrict__ gs,
                                               const int* __restrict__ colptr, const int4* __restrict__ ent_g,
                                               const int* __restrict__ shift, const int2* __restrict__ pixT, int ntx, const int* __restrict__ count,
                                               const uint2* __restrict__ list, double* __restrict__ L, int ldL,
                                               const double* __restrict__ svec, int* __restrict__ emax,
                                               unsigned char* __restrict__ nz, int nst)
{
    extern __shared__ __align__(16) int2 taps64[];  // [pnx + 62][pitch]: column pk + 31, row pl + R - 1
    constexpr int R = PSFX_R;
    const int pnx = sd.pnx, pny = sd.pny, nxh = pnx / 2, nyh = pny / 2, nxp = sd.nx + 2 * nxh;
    const int pitch = psfx_pitch(pny);
    const int lane = threadIdx.x & 31, nw = blockDim.x >> 5, items = *count;
    if ((int)blockIdx.x * nw >= items) return;
    if (FIXED) {
        for (int t = threadIdx.x; t < (pnx + 62) * pitch; t += blockDim.x) {
            const int pk = t / pitch - 31, pl = t % pitch - (R - 1);
            taps64[t] = (pk >= 0 && pk < pnx && pl >= 0 && pl < pny) ? sd.psf_fine[pl * pnx + pk] : make_int2(0, 0);
        }
        __syncthreads();
    }
    for (int it = blockIdx.x * nw + (threadIdx.x >> 5); it < items; it += gridDim.x * nw) {
        const uint2 item = list[it];
        const int s = item.x, y0 = (int)item.y / ntx * R, x0 = ((int)item.y % ntx) * 32, x = x0 + lane;
        const int n = colptr[s + 1] - colptr[s];
        const int4* ent = ent_g + colptr[s];
        int lo = 0, hi = n;
        if (n > 64) {
            lo = warp_lower_bound_row(ent, n, y0 + nyh - pny + 1);
            hi = warp_lower_bound_row(ent, n, y0 + R + nyh);
        }
        // th vh, th vl and tl vh: at most 2^62, 2^62 and 2^63 (StaticData::psf_w)
        long long hh[R], hl[R], lh[R];
        double acc[R];
        #pragma unroll
        for (int r = 0; r < R; r++) hh[r] = hl[r] = lh[r] = 0;
        #pragma unroll
        for (int r = 0; r < R; r++) acc[r] = 0;
        unsigned bad = 0;
        for (int e0 = lo; e0 < hi; e0 += 32) {
            int dx = -32, dy = 0, vh = 0, vl = 0;
            if (e0 + lane < hi) {
                const int4 en = ent[e0 + lane];
                dx = x0 - (ent_col(en) - nxh);           // column of lane 0's tap
                dy = y0 - (ent_row(en) - nyh);           // row of the first row's tap
                vh = en.y;
                vl = en.z;
            }
            unsigned hit = __ballot_sync(0xffffffffu, dx > -32 && dx < pnx && dy > -R && dy < pny);
            const unsigned nan = __ballot_sync(0xffffffffu, FIXED && vh == PSF64_BAD);
            for (; hit; hit &= hit - 1) {
                const int f = __ffs(hit) - 1;
                const int ox = __shfl_sync(0xffffffffu, dx, f) + lane, oy = __shfl_sync(0xffffffffu, dy, f);
                const int eh = __shfl_sync(0xffffffffu, vh, f), el = __shfl_sync(0xffffffffu, vl, f);
                if (nan >> f & 1) {
                    if (ox >= 0 && ox < pnx)
                        for (int r = 0; r < R; r++) bad |= (oy + r >= 0 && oy + r < pny) ? 1u << r : 0u;
                } else if (FIXED) {
                    const int2* tp = taps64 + (ox + 31) * pitch + oy + R - 1;
                    #pragma unroll
                    for (int r = 0; r < R; r++) {
                        const int2 t = tp[r];
                        hh[r] += (long long)t.x * eh;
                        hl[r] += (long long)t.x * el;
                        lh[r] += (long long)t.y * eh;
                    }
                } else if (ox >= 0 && ox < pnx) {
                    const double v = __hiloint2double(el, eh);
                    #pragma unroll
                    for (int r = 0; r < R; r++)
                        if (oy + r >= 0 && oy + r < pny) acc[r] = fma(sd.psf[ox * pny + oy + r], v, acc[r]);
                }
            }
        }
        int top = 0;
        if (x < sd.nx) {
            #pragma unroll
            for (int r = 0; r < R; r++) {
                if (y0 + r >= sd.ny) break;
                const int row = pixT[(size_t)(y0 + r + nyh) * nxp + x + nxh].x;
                if (row < 0) continue;
                double v = acc[r];
                if (FIXED) {
                    // as many of the lower halves' bits as there is room for
                    const int sh = max(0, min(min(20, sd.psf_w), __clzll(hh[r] < 0 ? -hh[r] : hh[r]) - 3));
                    v = fixed_to_double((hh[r] << sh) + (hl[r] >> (29 - sh)) + (lh[r] >> (sd.psf_w - sh)),
                                        sd.psf_t + 28 + sh + shift[s]);
                }
                if (bad >> r & 1) v = __longlong_as_double(0x7ff8000000000000ll);
                const int e = exponent_of(v);
                if (e == 0) continue;
                L[(size_t)s * ldL + row] = v;
                nz[(size_t)(s / 64) * nst + row / 32] = 1;
                top = max(top, svec ? exponent_of(v * svec[row]) : e);
            }
        }
        for (int o = 16; o > 0; o >>= 1) top = max(top, __shfl_xor_sync(0xffffffffu, top, o));
        if (lane == 0 && top > 0) atomicMax(&emax[s], top);
    }
}

// Active row -> image pixel, the inverse of the compaction's pixindex, and the
// row's data and C^-1 (svec, or null: the root of its size, with its sign).
__global__ void k_rowpix(StaticData sd_, const int* __restrict__ rowidx, int* __restrict__ rowpix,
                         double* __restrict__ dvec, double* __restrict__ cvec, double* __restrict__ svec)
{
    const StaticData sd = eval_shape(sd_);
    for (int m = blockIdx.x * blockDim.x + threadIdx.x; m < sd.n_mask; m += gridDim.x * blockDim.x) {
        const int r = rowidx[m];
        if (r < 0) continue;
        const int pix = sd.mpix[m];
        rowpix[r] = pix;
        dvec[r] = sd.data[pix];
        cvec[r] = sd.use_noise_map ? sd.covinv[pix] : sd.cov_inverse;
        if (svec) svec[r] = cvec[r] < 0 ? -sqrt(-cvec[r]) : sqrt(cvec[r]);
    }
}

void psf_init_attributes()
{
    cudaFuncSetAttribute(k_psf64<true>, cudaFuncAttributeMaxDynamicSharedMemorySize, PSF64_PAD_BYTES);
}

void launch_rowpix(const StaticData& sd, Work& w, cudaStream_t st)
{
    if (sd.n_mask == 0) return;
    k_rowpix<<<(sd.n_mask + 255) / 256, 256, 0, st>>>(sd, w.rowidx, w.rowpix, w.dvec, w.cvec,
                                                        sd.use_noise_map ? w.svec : nullptr);
    count_launches(1);
}

// The plain path's stated range of PSFs and source grids: calls past it were refused by its
// first kernel, which held a row of L' and the taps in shared memory, and stay refused
// (k_psf64 itself would take them).
int psf_in_range(const StaticData& sd, int M_max)
{
    const size_t nT = ((size_t)sd.pnx * sd.pny + 7) / 8 * 8;
    if (8 * (M_max + nT) + 8 * nT <= 227 * 1024) return QLP_OK;
    set_error("%s (%d)", "PSF and source grid too large for the plain path", (int)nT);
    return QLP_ERR_CUDA;
}

void launch_psf(const StaticData& sd, Work& w, int N_max, cudaStream_t st)
{
    if (N_max == 0) return;
    const size_t taps = sizeof(int2) * psfx_taps(sd.pnx, sd.pny);
    const bool fixed = sd.psf_fixed && taps <= PSF64_PAD_BYTES;
    w.csc.raw = fixed ? 0 : 1;
    launch_csc(sd, w, w.csc, N_max, w.Lpsf, w.ldL, st);
    auto k = fixed ? k_psf64<true> : k_psf64<false>;
    k<<<152 * 3, 256, fixed ? taps : 0, st>>>(sd, w.gs, w.csc.colcnt, w.csc.fine, w.csc.shift, w.csc.pixT,
                                            (sd.nx + 31) / 32,
                                            w.csc.ntiles(), w.csc.tiles, w.Lpsf, w.ldL, sd.use_noise_map ? w.svec : nullptr,
                                            oz_emax(w.oz), oz_nz(w.oz), oz_nst(w.oz));
    count_launches(1);
}

}  // namespace qlpix
