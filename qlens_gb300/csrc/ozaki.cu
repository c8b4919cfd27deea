// ozaki.cu -- the plain path's FP64 contraction F = L'^T C^-1 L' on the tensor
// cores: L' cut into digits (k_oz_slice), the digit products
// (k_oz_syrk, ozaki.cuh) and the integers turned into F (k_oz_finish).
// Reference: QLens::create_lensing_matrices_from_Lmatrix_dense
// (pixelgrid.cpp:15590-15736).
#include <cuda_fp16.h>
#include <algorithm>
#include "qlpix_ctx.h"
#include "ozaki.cuh"
#include "tma_map.h"

namespace qlpix {

#define OZ_S 7                      // digits of L' (54 bits)

// Digits of L' kept at a time: a larger L' goes in chunks of image pixels, the
// integer sums of the chunks adding up.
#define OZ_CHUNK_BYTES ((size_t)1 << 30)
// Digit products in flight: with fewer tiles than this the pixels of each tile
// are split over several CTAs (one CTA per SM; two rounds even out the sparsity)
#define OZ_WANT_CTAS (2 * 152)

struct OzWork {
    __half* xs = nullptr;              // [OZ_S][M128][Kc] digits of L'^T sqrt(C^-1)
    unsigned long long* part = nullptr; // [tile][hi, lo][64 columns][128 rows], zero between evaluations
    int* emax = nullptr;               // [M128] largest biased exponent of each source cell's L' (sqrt(C^-1))
    unsigned char* nz = nullptr;       // [M128 / 64][nst] 32-pixel stages where 64 cells have a nonzero
    int M128 = 0, Kc = 0, nst = 0, ntiles = 0;
    CUtensorMap map_a, map_b;
};

// Tile t of the lower triangle: 128-row block I, 64-column block j <= 2 I + 1.
__device__ __forceinline__ void oz_tile(int t, int& I, int& j)
{
    int i = (int)((sqrtf(4.0f * t + 1.0f) - 1.0f) * 0.5f);
    while ((i + 1) * (i + 2) <= t) i++;
    while (i * (i + 1) > t) i--;
    I = i;
    j = t - i * (i + 1);
}

// The digits of 64 cells x 32 pixels of L'^T (sqrt(C^-1)), eight pixels a thread.  With a
// noise map the operand is the product L' sqrt(C^-1) as k_psf64 formed it for the cell's
// largest exponent (a bound from the image's largest sqrt(C^-1) instead cost a cell on
// noisier pixels as many of its bits as their noise is larger).  sign: the pixels with
// this sign of C^-1.
// Stages without a nonzero in the cells' 128-row block are never loaded by the
// products, so they are skipped.  14 bytes written per 8 read: DRAM at 70 % of its measured
// rate (75 us at 2,934 cells x 11,772 pixels).
__global__ void __launch_bounds__(256) k_oz_slice(const GridState* __restrict__ gs, const double* __restrict__ L,
                                                  int ldL, const double* __restrict__ svec, int sign,
                                                  const int* __restrict__ emax, const unsigned char* __restrict__ nz,
                                                  int nst, int st0, __half* __restrict__ xs, int M128, int Kc)
{
    const int N = gs->N, M = gs->M;
    const int cb = blockIdx.y, st = st0 + blockIdx.x;
    const int ncb = (M + 63) / 64;
    if (cb >= ((ncb + 1) & ~1) || st * 32 >= N) return;
    const int other = cb ^ 1;
    const bool live = cb < ncb && nz[(size_t)cb * nst + st];
    if (!(live || (other < ncb && nz[(size_t)other * nst + st]))) return;
    const int c = threadIdx.x >> 2, k0 = (threadIdx.x & 3) * 8, cell = cb * 64 + c, r0 = st * 32 + k0;
    unsigned long long q[8];
    #pragma unroll
    for (int u = 0; u < 8; u++) q[u] = oz_bias<OZ_S>(0);
    const int em = (cell < M) ? emax[cell] : 0;
    if (live && em > 0 && em < 2047) {
        #pragma unroll
        for (int u = 0; u < 8; u += 2) {
            const double2 v = *reinterpret_cast<const double2*>(L + (size_t)cell * ldL + r0 + u);
            #pragma unroll
            for (int k = 0; k < 2; k++) {
                const int r = r0 + u + k;
                double x = r < N ? (k ? v.y : v.x) : 0.0;
                if (svec && x != 0) x = (svec[r] < 0) == (sign < 0) ? x * fabs(svec[r]) : 0.0;
                q[u + k] = oz_bias<OZ_S>(oz_fixed54(x, em));
            }
        }
    }
    __half* out = xs + (size_t)cell * Kc + (size_t)blockIdx.x * 32 + k0;
    #pragma unroll
    for (int d = 0; d < OZ_S; d++) {
        *reinterpret_cast<uint4*>(out + (size_t)d * M128 * Kc) = oz_digits8<OZ_S>(q, d);
    }
}

// What bounds it: the tensor pipe where a stage is live, 28 digit products of
// 128 x 64 x 32 each (an N = 64 MMA reads 6 KB of shared memory per 32 clocks of
// arithmetic, so it runs at about two thirds of the pipe), and the reading of
// the accumulators beside it.  The FP64 pipe's SYRK that it replaces (64x64
// tiles, the same zero blocks skipped) was at 99 % of that pipe: F of 2,934
// cells x 11,772 pixels 23.5 -> 1.10 ms, 738 x 6,220 4.29 -> 0.13 ms, 96 x 448
// 0.48 -> 0.05 ms, everything of launch_syrk_fp64 included.
// The digit products of one tile over its share of the chunk's live stages
// (both blocks have a nonzero among the stage's 32 pixels): grid (tiles,
// splits).  The tile's integers are added into `part` (sign < 0: taken off) by 64-bit
// reductions, lanes along the rows.
__global__ void __launch_bounds__(OZ_THREADS, 1) k_oz_syrk(const __grid_constant__ CUtensorMap map_a,
                                                          const __grid_constant__ CUtensorMap map_b, GridState* gs,
                                                          const unsigned char* __restrict__ nz, int nst, int st0,
                                                          int st1, int M128, unsigned long long* __restrict__ part,
                                                          int sign)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ OzPipe pipe;
    __shared__ int n_live;
    int I, j;
    oz_tile(blockIdx.x, I, j);
    const int ncb = (gs->M + 63) / 64;
    if (j >= ncb || 2 * I >= ncb) return;
    const unsigned char* fa = nz + (size_t)(2 * I) * nst;
    const unsigned char* fb = (2 * I + 1 < ncb) ? fa + nst : fa;      // the block's second 64 rows, if there are any
    const unsigned char* fj = nz + (size_t)j * nst;
    const int e = min(st1, (gs->N + 31) >> 5);
    if (threadIdx.x == 0) n_live = 0;
    __syncthreads();
    int cnt = 0;
    for (int k = st0 + threadIdx.x; k < e; k += blockDim.x) cnt += ((fa[k] | fb[k]) & fj[k]) ? 1 : 0;
    if (cnt) atomicAdd(&n_live, cnt);
    __syncthreads();
    const int total = n_live;
    const int s0 = (int)((long long)total * blockIdx.y / gridDim.y);
    const int n = (int)((long long)total * (blockIdx.y + 1) / gridDim.y) - s0;     // this CTA's live stages
    if (n == 0) return;

    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    oz_begin(pipe);
    long long hi[32];
    uint32_t lo[32];
    bool ok = true;
    if (warp == OZ_EPI) {
        // TMA: 32 stages' flags at a time, the live ones in order
        int seen = 0, it = 0;
        bool good = true;
        for (int k0 = st0; k0 < e && it < n && good; k0 += 32) {
            const int k = k0 + lane;
            unsigned live = __ballot_sync(0xffffffffu, k < e && ((fa[k] | fb[k]) & fj[k]));
            const int c = __popc(live);
            if (seen + c <= s0) { seen += c; continue; }
            for (; live && it < n; live &= live - 1) {
                if (seen++ < s0) continue;
                const int st = k0 + __ffs(live) - 1;
                if (lane == 0) {
                    good = good && oz_load_stage<OZ_S>(pipe, smem, it, &map_a, &map_b, M128, (st - st0) * 32, I * OZ_TM,
                                                 j * OZ_TN);
                    if (good) pipe.n_issued = it + 1;
                }
                it++;
            }
            good = __shfl_sync(0xffffffffu, good, 0);
        }
    } else if (warp == OZ_EPI + 1) {
        if (lane == 0) {
            oz_mma_loop<OZ_S>(pipe, smem, 0, 0, n);
            mma_commit(&pipe.done);
        }
    } else {
        #pragma unroll
        for (int c = 0; c < 32; c++) hi[c] = lo[c] = 0;
        ok = oz_accumulate<OZ_S>(pipe, 0, n, hi, lo);
    }
    __syncwarp();
    oz_end(pipe);
    if (pipe.abort) {
        if (threadIdx.x == 0) atomicExch(&gs->status, QLP_ERR_TIMEOUT);
        return;
    }
    if (warp < OZ_EPI && ok) {
        unsigned long long* out = part + (size_t)blockIdx.x * 2 * OZ_TM * OZ_TN + (size_t)(warp >> 2) * 32 * OZ_TM +
                                  (warp & 3) * 32 + lane;
        #pragma unroll
        for (int c = 0; c < 32; c++) {
            atomicAdd(out + c * OZ_TM, (unsigned long long)(sign < 0 ? -hi[c] : hi[c]));
            atomicAdd(out + OZ_TM * OZ_TN + c * OZ_TM,
                      sign < 0 ? 0ull - (unsigned long long)lo[c] : (unsigned long long)lo[c]);
        }
    }
}

// F from the integers: (hi 2^24 + lo) 2^(Ea + Eb - 60) times the uniform C^-1,
// and the integers set back to zero.  A CTA takes 32 columns of a tile, through
// shared memory so that both sides move whole rows.
__global__ void __launch_bounds__(256) k_oz_finish(const GridState* __restrict__ gs,
                                                   unsigned long long* __restrict__ part,
                                                   const int* __restrict__ emax, double scale,
                                                   double* __restrict__ F, int ldF)
{
    __shared__ double s[32][OZ_TM + 1];
    int I, j;
    oz_tile(blockIdx.x >> 1, I, j);
    const int h = blockIdx.x & 1;
    const int M = gs->M, Mp = (M + 63) & ~63;
    if (I * OZ_TM >= Mp || j * OZ_TN >= Mp) return;
    unsigned long long* in = part + (size_t)(blockIdx.x >> 1) * 2 * OZ_TM * OZ_TN + (size_t)h * 32 * OZ_TM;
    const int r = threadIdx.x & 127, a = I * OZ_TM + r;
    const double sa = (a < M) ? oz_scale(emax[a]) : 0.0;
    for (int c = threadIdx.x >> 7; c < 32; c += 2) {
        const long long hi = (long long)in[c * OZ_TM + r], lo = (long long)in[OZ_TM * OZ_TN + c * OZ_TM + r];
        in[c * OZ_TM + r] = 0;
        in[OZ_TM * OZ_TN + c * OZ_TM + r] = 0;
        const int b = j * OZ_TN + h * 32 + c;
        const double sb = (b < M) ? oz_scale(emax[b]) : 0.0;
        // 2^-60 split over the two scales' products: no overflow on the way
        s[c][r] = ((fma((double)hi, 16777216.0, (double)lo) * 0x1p-60 * sa) * sb) * scale;
    }
    __syncthreads();
    const int c = threadIdx.x & 31;
    for (int row = threadIdx.x >> 5; row < OZ_TM; row += 8)
        if (I * OZ_TM + row < Mp) F[(size_t)(I * OZ_TM + row) * ldF + j * OZ_TN + h * 32 + c] = s[c][row];
}

void oz_free(OzWork* z)
{
    if (!z) return;
    void* ptrs[] = {z->xs, z->part, z->emax, z->nz};
    for (void* p : ptrs) if (p) cudaFree(p);
    delete z;
}

// Workspace for N_cap image pixels and M_cap source cells.
int oz_alloc(OzWork** out, int N_cap, int M_cap)
{
    OzWork* z = new OzWork();
    z->M128 = (M_cap + OZ_TM - 1) / OZ_TM * OZ_TM;
    const int nI = z->M128 / OZ_TM;
    z->ntiles = nI * (nI + 1);
    z->nst = (std::max(N_cap, 1) + 31) / 32;
    const int fit = (int)std::min<size_t>(1u << 20, OZ_CHUNK_BYTES / ((size_t)OZ_S * 2 * z->M128)) / 128 * 128;
    z->Kc = std::min(z->nst * 32, std::max(128, fit));
    cudaError_t e = cudaSuccess;
    auto A = [&](void** p, size_t bytes) { if (e == cudaSuccess) e = cudaMalloc(p, bytes); };
    const size_t pbytes = (size_t)z->ntiles * 2 * OZ_TM * OZ_TN * sizeof(long long);
    // the factorisation of F keeps its digits (eight of M128 columns) in the same buffer
    A((void**)&z->xs, sizeof(__half) * (size_t)z->M128 * std::max(OZ_S * z->Kc, 8 * z->M128));
    A((void**)&z->part, pbytes);
    A((void**)&z->emax, sizeof(int) * z->M128);
    A((void**)&z->nz, (size_t)(z->M128 / 64) * z->nst + 3);
    if (e == cudaSuccess) e = cudaMemset(z->part, 0, pbytes);
    if (e == cudaSuccess) e = cudaStreamSynchronize(0);    // the slots' streams do not wait for stream 0
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_oz_syrk, cudaFuncAttributeMaxDynamicSharedMemorySize, oz_smem(OZ_S));
    int rc = QLP_OK;
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("%s (%d)", "FP64 contraction workspace", (int)e);
        rc = (e == cudaErrorMemoryAllocation) ? QLP_ERR_NOMEM : QLP_ERR_CUDA;
    } else if (make_map_box(&z->map_a, z->xs, (size_t)OZ_S * z->M128, z->Kc, true, OZ_TM, OZ_KS) != QLP_OK ||
               make_map_box(&z->map_b, z->xs, (size_t)OZ_S * z->M128, z->Kc, true, OZ_TN, OZ_KS) != QLP_OK) {
        set_error("%s (%d)", "cuTensorMapEncodeTiled unavailable or failed", 0);
        rc = QLP_ERR_CUDA;
    }
    if (rc != QLP_OK) { oz_free(z); return rc; }
    *out = z;
    return QLP_OK;
}

void oz_clear(const OzWork* z, ClearList& l)
{
    l.add(z->emax, sizeof(int) * z->M128);
    l.add(z->nz, (size_t)(z->M128 / 64) * z->nst);
}

// What the build of L' (k_psf64) fills in: each cell's largest exponent and the
// live 32-pixel stages of each 64 cells.
int* oz_emax(OzWork* z) { return z->emax; }
unsigned char* oz_nz(OzWork* z) { return z->nz; }
int oz_nst(const OzWork* z) { return z->nst; }

// The digits' buffer, free once F stands.
void* oz_buffer(OzWork* z) { return z->xs; }

void launch_syrk_fp64(const StaticData& sd, Work& w, int N_max, int M_max, cudaStream_t st)
{
    OzWork* z = w.oz;
    const int nI = (M_max + OZ_TM - 1) / OZ_TM, tiles = nI * (nI + 1), ncb = 2 * nI;
    int n = 0;
    const int nst = (N_max + 31) / 32, per = z->Kc / 32;
    for (int s0 = 0; s0 < nst; s0 += per) {
        const int cnt = std::min(per, nst - s0);
        // pixels split so that a small problem's few tiles still fill the GPU,
        // but no finer than one read of the accumulators per CTA
        const int split = std::max(1, std::min({(OZ_WANT_CTAS + tiles - 1) / tiles, (cnt + OZ_FLUSH - 1) / OZ_FLUSH,
                                                64}));
        // (a noise map with negative C^-1, no one's noise but taken: those pixels in a turn of their own)
        for (int sign = 1; sign >= (sd.neg_noise ? -1 : 1); sign -= 2) {
            k_oz_slice<<<dim3(cnt, ncb), 256, 0, st>>>(w.gs, w.Lpsf, w.ldL, sd.use_noise_map ? w.svec : nullptr, sign,
                                                       z->emax, z->nz, z->nst, s0, z->xs, z->M128, z->Kc);
            k_oz_syrk<<<dim3(tiles, split), OZ_THREADS, oz_smem(OZ_S), st>>>(z->map_a, z->map_b, w.gs, z->nz, z->nst,
                                                                       s0, s0 + cnt, z->M128, z->part, sign);
            n += 2;
        }
    }
    k_oz_finish<<<2 * tiles, 256, 0, st>>>(w.gs, z->part, z->emax, sd.use_noise_map ? 1.0 : sd.cov_inverse, w.F,
                                           w.ldF);
    count_launches(n + 1);
}

}  // namespace qlpix
