// chol128.cuh -- FP32 Cholesky of the mixed path, 128-column blocks, one launch
// per matrix.
//
// Left-looking: CTAs take 128x128 tiles, column by column, from a counter.  A
// tile (i, j) subtracts L_ik L_jk^T over the finished columns k < j: TMA loads of
// the split factor (F16 hi + lo, each row of a block scaled by a power of two
// near 2^14; 64-column boxes, 128-byte swizzle), three products hi*hi + hi*lo +
// lo*hi of tcgen05 kind::f16 (~22 significant bits), the accumulators in two TMEM
// buffers, each column block's product subtracted in FP32 registers with its
// scales undone exactly while the next one's MMAs run.  Then
//   i = j   the block is factored and inverted in shared memory (potrf128: four
//           32-column panels, a warp's register Cholesky for the 32x32 piece, the
//           rows below one per thread, the trailing piece in 4x4 register blocks;
//           the inverse's 32x32 blocks by distance) and the inverse is published
//           split into TF32 hi + lo;
//   i > j   L_ij = A_ij L_jj^-T by 3xTF32 products with that inverse, published as
//           F16 hi + lo for the tiles to come and in FP32 for the solves.
// A tile waits by flags on tiles with a smaller number only, which are finished
// or held by running CTAs, so any grid size works; every wait is bounded (~1 s).
// The operations and their order are those of the right-looking version that
// this replaces (three launches per step, 188 an evaluation at a capacity of
// 4,096 cells, most of them empty for a smaller grid; every trailing tile read
// and written once per step), so the results are the same but
// for a last digit now and then.  Bound by the
// chain of pivot blocks: 66 us a column, 46 of them the block (11 its inverse) and
// 20 from its end to the next diagonal tile's start; 4,096 cells with the solves
// 2.6 -> 2.0 ms.
// `band`: blocks below the diagonal that can be nonzero: the curvature matrix R
// couples a cell only to cells at most two grid rows away.
// QLens factors with Cholesky_dcmp_packed (pixelgrid.cpp:17071-17105): a
// negative pivot is recorded and sqrt(|d|) used; the first such pivot is
// reported through GridState::not_spd_F / not_spd_R.
#pragma once
#include <cuda_fp16.h>
#include "tc_common.cuh"

namespace qlpix {

#define C2 128
#define C2_STAGES 3
#define C2_STAGE_BYTES (4 * TC_TILE_BYTES)                // [A/B][hi/lo] of 64 columns
#define C2_SMEM (C2_STAGES * C2_STAGE_BYTES + 1024)
#define C2_EPI 8                                          // epilogue warps
#define C2_THREADS (32 * (C2_EPI + 2))                    // + TMA and MMA warps

__device__ __forceinline__ int cpad128(int M) { return (M + C2 - 1) / C2 * C2; }

__device__ __forceinline__ void tri_ij(int t, int& i, int& j)
{
    i = (int)((sqrtf(8.0f * t + 1.0f) - 1.0f) * 0.5f);   // corrected below
    while ((i + 1) * (i + 2) / 2 <= t) i++;
    while (i * (i + 1) / 2 > t) i--;
    j = t - i * (i + 1) / 2;
}

// One step of the register Cholesky of a 32x32 block held one row per lane
// (lane l: a[c] = L[l][c], entries right of the diagonal are not kept);
// unrolled at compile time so a[] stays in registers.  The finished column
// goes round through shared memory (buf: 2 x 32 floats, alternating), 128-bit
// broadcasts; only the next pivot's factor comes by a shuffle, so that the
// chain from pivot to pivot is two shuffles and an rsqrt (all of them by
// shuffles had the shuffle unit bound it).
template <int J>
__device__ __forceinline__ void warp_chol32(float (&a)[32], int lane, int& bad, float* buf)
{
    if constexpr (J < 32) {
        const float d = __shfl_sync(0xffffffffu, a[J], J);
        bad = (d < 0.f && bad == 0) ? J + 1 : bad;      // the first negative pivot
        const float rs = rsqrtf(fabsf(d));      // FP32 path: 1/sqrt and a multiply, not sqrt and a divide
        a[J] = (lane == J ? fabsf(d) : a[J]) * rs;
        if constexpr (J < 30) buf[(J & 1) * 32 + lane] = a[J];
        if constexpr (J < 31) a[J + 1] -= a[J] * __shfl_sync(0xffffffffu, a[J], J + 1);
        __syncwarp();
        const float4* col = reinterpret_cast<const float4*>(buf + (J & 1) * 32);
        #pragma unroll
        for (int q = (J + 2) / 4; q < 8; q++) {
            const float4 v = col[q];
            if (4 * q > J + 1) a[4 * q] -= a[J] * v.x;
            if (4 * q + 1 > J + 1) a[4 * q + 1] -= a[J] * v.y;
            if (4 * q + 2 > J + 1) a[4 * q + 2] -= a[J] * v.z;
            if (4 * q + 3 > J + 1) a[4 * q + 3] -= a[J] * v.w;
        }
        warp_chol32<J + 1>(a, lane, bad, buf);
    }
}

// barrier of the first 256 threads
__device__ __forceinline__ void c2_sync() { asm volatile("bar.sync 1, 256;" ::: "memory"); }

__device__ __forceinline__ float2 split_tf32(float x)
{
    uint32_t h, l;
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h) : "f"(x));
    asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l) : "f"(x - __uint_as_float(h)));
    return make_float2(__uint_as_float(h), __uint_as_float(l));
}

// The B x B block (i0, j0) of the lower triangle less the panel's product: S -= P P^T
// over the 32 columns from c0.
template <int B>
__device__ __forceinline__ void potrf_trail(float (*S)[C2 + 1], int i0, int j0, int c0)
{
    float acc[B][B];
    #pragma unroll
    for (int u = 0; u < B; u++)
        #pragma unroll
        for (int v = 0; v < B; v++) acc[u][v] = 0.f;
    #pragma unroll 8
    for (int m = 0; m < 32; m++) {
        float ra[B], rb[B];
        #pragma unroll
        for (int u = 0; u < B; u++) { ra[u] = S[i0 + u][c0 + m]; rb[u] = S[j0 + u][c0 + m]; }
        #pragma unroll
        for (int u = 0; u < B; u++)
            #pragma unroll
            for (int v = 0; v < B; v++) acc[u][v] += ra[u] * rb[v];
    }
    #pragma unroll
    for (int u = 0; u < B; u++)
        #pragma unroll
        for (int v = 0; v < B; v++)
            if (j0 + v <= i0 + u) S[i0 + u][j0 + v] -= acc[u][v];
}

// Inverse of the 32x32 diagonal block at b0 by one warp, lane = column.
__device__ __forceinline__ void potrf_inv32(float (*S)[C2 + 1], float (*V)[C2 + 1], const float* rdiag, int b0, int lane)
{
    float x[32];
    #pragma unroll
    for (int i = 0; i < 32; i++) {
        float acc = (i == lane) ? 1.f : 0.f;
        #pragma unroll
        for (int m = 0; m < i; m++) acc -= S[b0 + i][b0 + m] * x[m];
        x[i] = (i < lane) ? 0.f : acc * rdiag[b0 + i];
    }
    #pragma unroll
    for (int i = 0; i < 32; i++) V[b0 + i][b0 + lane] = x[i];
}

// The 128x128 block at the head of p128_smem (rows of 129, upper part zero),
// factored and inverted by the first 256 threads; the inverse split into TF32
// hi + lo goes to ih, il.  o: the block's first pivot (for the flag).
// What bounds it is one SM's chain of 128 pivots and its shared-memory reads: a
// warp factors each 32x32 piece in registers while the other warps update the
// rest of the trailing block (it updates the next piece itself first), the
// pieces' inverses run beside the row solves, and the inverse's off-diagonal
// blocks are formed in 4x4 register blocks (one product per read had made them a
// third of the time).  Each entry's operations and their order are those of the
// plain blocked algorithm.
__device__ __forceinline__ void potrf128(float* p128_smem, int o, int* flag, float* __restrict__ ih,
                                         float* __restrict__ il)
{
    float (*S)[C2 + 1] = reinterpret_cast<float (*)[C2 + 1]>(p128_smem);
    float (*V)[C2 + 1] = reinterpret_cast<float (*)[C2 + 1]>(p128_smem + C2 * (C2 + 1));
    float* rdiag = p128_smem + 2 * C2 * (C2 + 1);         // 1 / L_ii
    float* buf = rdiag + C2;                              // warp 0's column buffer
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    auto factor32 = [&](int c0) {
        float a[32];
        #pragma unroll
        for (int c = 0; c < 32; c++) a[c] = S[c0 + lane][c0 + c];
        int bad = 0;
        warp_chol32<0>(a, lane, bad, buf);
        if (lane == 0 && bad != 0 && *flag == 0) *flag = o + c0 + bad;
        #pragma unroll
        for (int c = 0; c < 32; c++) {
            S[c0 + lane][c0 + c] = (c <= lane) ? a[c] : 0.f;
            if (c == lane) rdiag[c0 + lane] = 1.0f / a[c];
        }
    };
    if (warp == 0) factor32(0);
    c2_sync();
    #pragma unroll 1
    for (int p = 0; p < 3; p++) {
        const int c0 = p * 32, t0 = c0 + 32, below = C2 - t0;
        if (tid < below) {                       // rows below: x L_pp^T = a
            const int r = t0 + tid;
            float x[32];
            #pragma unroll
            for (int c = 0; c < 32; c++) x[c] = S[r][c0 + c];
            #pragma unroll
            for (int c = 0; c < 32; c++) {
                float a0 = x[c], a1 = 0.f;
                #pragma unroll
                for (int m = 0; m + 1 < c; m += 2) {
                    a0 -= x[m] * S[c0 + c][c0 + m];
                    a1 -= x[m + 1] * S[c0 + c][c0 + m + 1];
                }
                if (c & 1) a0 -= x[c - 1] * S[c0 + c][c0 + c - 1];
                x[c] = (a0 + a1) * rdiag[c0 + c];
            }
            #pragma unroll
            for (int c = 0; c < 32; c++) S[r][c0 + c] = x[c];
        } else if (warp == 7) {
            potrf_inv32(S, V, rdiag, c0, lane);
        }
        c2_sync();
        // trailing lower triangle: the next 32x32 piece in 2x2 blocks by four
        // warps, then its factorisation in warp 0 while the others do the rest in
        // 4x4 blocks
        const int nb = below / 4, nblk = nb * (nb + 1) / 2;
        if (warp < 4) {
            for (int b = tid; b < 136; b += 128) {
                int bi, bj;
                tri_ij(b, bi, bj);
                potrf_trail<2>(S, t0 + 2 * bi, t0 + 2 * bj, c0);
            }
            asm volatile("bar.sync 3, 128;" ::: "memory");
        }
        if (warp == 0) {
            factor32(t0);
        } else {
            for (int b = 36 + 255 - tid; b < nblk; b += 224) {
                int bi, bj;
                tri_ij(b, bi, bj);
                potrf_trail<4>(S, t0 + 4 * bi, t0 + 4 * bj, c0);
            }
        }
        c2_sync();
    }
    // ---- off-diagonal blocks of V = L^-1 by distance d: V_ij = -V_ii (sum_{k=j}^{i-1} L_ik V_kj) ----
    // The blocks of one distance depend only on nearer ones, so all of them are
    // formed together.  The products sum_k L_ik V_kj go into the upper triangle
    // of V (block (j, i)), which nothing reads as V; those of distance 1 do not
    // need the last diagonal block's inverse, which is formed beside them.
    #pragma unroll 1
    for (int d = 1; d < 4; d++) {
        const int jb = tid >> 6, ib = jb + d, r = (tid >> 1) & 28, c = (tid & 7) * 4;
        const bool mine = tid < (4 - d) * 64;
        float acc[4][4];
        if (d == 1 && warp == 7) potrf_inv32(S, V, rdiag, 96, lane);
        if (mine) {
            #pragma unroll
            for (int u = 0; u < 4; u++)
                #pragma unroll
                for (int v = 0; v < 4; v++) acc[u][v] = 0.f;
            const int m1 = ib * 32;
            #pragma unroll 8
            for (int m = jb * 32; m < m1; m++) {
                float ra[4], rb[4];
                #pragma unroll
                for (int u = 0; u < 4; u++) { ra[u] = S[ib * 32 + r + u][m]; rb[u] = V[m][jb * 32 + c + u]; }
                #pragma unroll
                for (int u = 0; u < 4; u++)
                    #pragma unroll
                    for (int v = 0; v < 4; v++) acc[u][v] += ra[u] * rb[v];
            }
            #pragma unroll
            for (int u = 0; u < 4; u++)
                #pragma unroll
                for (int v = 0; v < 4; v++) V[jb * 32 + r + u][ib * 32 + c + v] = acc[u][v];
        }
        c2_sync();
        if (mine) {
            #pragma unroll
            for (int u = 0; u < 4; u++)
                #pragma unroll
                for (int v = 0; v < 4; v++) acc[u][v] = 0.f;
            #pragma unroll 4
            for (int m = 0; m < r + 4; m++) {    // (V_ii is zero above its diagonal)
                float ra[4], rb[4];
                #pragma unroll
                for (int u = 0; u < 4; u++) { ra[u] = V[ib * 32 + r + u][ib * 32 + m]; rb[u] = V[jb * 32 + m][ib * 32 + c + u]; }
                #pragma unroll
                for (int u = 0; u < 4; u++)
                    #pragma unroll
                    for (int v = 0; v < 4; v++) acc[u][v] += ra[u] * rb[v];
            }
            #pragma unroll
            for (int u = 0; u < 4; u++)
                #pragma unroll
                for (int v = 0; v < 4; v++) V[ib * 32 + r + u][jb * 32 + c + v] = -acc[u][v];
        }
        c2_sync();
    }
    // the inverse's split (upper part zero), which the tiles below wait for
    #pragma unroll 4
    for (int u = 0; u < 16; u++) {
        const int idx = tid + u * 256, r = idx >> 5, c = (idx & 31) * 4;
        float2 v[4];
        #pragma unroll
        for (int e = 0; e < 4; e++) v[e] = split_tf32(c + e <= r ? V[r][c + e] : 0.f);
        *reinterpret_cast<float4*>(ih + (size_t)r * C2 + c) = make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
        *reinterpret_cast<float4*>(il + (size_t)r * C2 + c) = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
    }
}

// What nothing in the factorisation waits for: the factor's block to A, its
// inverse (row-major, upper part zero) and the inverse's transpose to Linv.
__device__ __forceinline__ void potrf128_store(float* p128_smem, float* __restrict__ A, int ld, float* __restrict__ Linv)
{
    float (*S)[C2 + 1] = reinterpret_cast<float (*)[C2 + 1]>(p128_smem);
    float (*V)[C2 + 1] = reinterpret_cast<float (*)[C2 + 1]>(p128_smem + C2 * (C2 + 1));
    const int tid = threadIdx.x;
    #pragma unroll 4
    for (int u = 0; u < 16; u++) {   // the factor (upper part of the block zero)
        const int idx = tid + u * 256, r = idx >> 5, c = (idx & 31) * 4;
        *reinterpret_cast<float4*>(A + (size_t)r * ld + c) =
            make_float4(S[r][c], S[r][c + 1], S[r][c + 2], S[r][c + 3]);
    }
    if (Linv == nullptr) return;
    #pragma unroll 4
    for (int u = 0; u < 16; u++) {
        const int idx = tid + u * 256, r = idx >> 5, c = (idx & 31) * 4;
        *reinterpret_cast<float4*>(Linv + (size_t)r * C2 + c) =
            make_float4(c <= r ? V[r][c] : 0.f, c + 1 <= r ? V[r][c + 1] : 0.f, c + 2 <= r ? V[r][c + 2] : 0.f,
                        c + 3 <= r ? V[r][c + 3] : 0.f);
        *reinterpret_cast<float4*>(Linv + C2 * C2 + (size_t)r * C2 + c) =
            make_float4(r <= c ? V[c][r] : 0.f, r <= c + 1 ? V[c + 1][r] : 0.f, r <= c + 2 ? V[c + 2][r] : 0.f,
                        r <= c + 3 ? V[c + 3][r] : 0.f);
    }
}

struct Flow128 {
    uint64_t full[C2_STAGES], empty[C2_STAGES];
    uint64_t acc_full[2], acc_empty[2], exp_full[2];      // per accumulator buffer; exp: the rows' scales
    uint64_t b_full, sol[2], done;
    uint32_t tmem;
    int n_issued, n_used, n_exp;                          // stages loaded / consumed, scales loaded
    volatile int abort;
};

// Untiled bulk copy to shared memory (16-byte aligned, a multiple of 16 bytes).
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

__device__ __forceinline__ void c2_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

__device__ __forceinline__ bool c2_wait_flag(const int* p, GridState* gs, volatile int* abort_flag)
{
    if (ld_acquire(p)) return true;
    const uint64_t t0 = globaltimer();
    while (!ld_acquire(p)) {
        if (*abort_flag || *(volatile int*)&gs->status == QLP_ERR_TIMEOUT || globaltimer() - t0 > TC_WAIT_NS) {
            *abort_flag = 1;
            return false;
        }
        __nanosleep(32);
    }
    return true;
}

// The factorisation's arrays: the split factor Lh, Ll [rows][128 wb], block column k at k
// mod wb (all of them, or of a band's rows the band + 1 that are still read), with each
// column block's row scales pexp[block][rows], the split inverses [rows][128]
// and the flags: ready[column][row block], inverse[column], tile counter.
struct Flow128Mem {
    __half* Lh;
    __half* Ll;
    int* pexp;
    float* ih;
    float* il;
    int* flags;
    int rows, wb;                                         // M_cap, a multiple of 128
};

__global__ void __launch_bounds__(C2_THREADS, 1) k_chol128(const __grid_constant__ CUtensorMap map_hi,
                                                          const __grid_constant__ CUtensorMap map_lo,
                                                          const __grid_constant__ CUtensorMap map_ih,
                                                          const __grid_constant__ CUtensorMap map_il, float* A, int ld,
                                                          GridState* gs, int which, int band, Flow128Mem mem,
                                                          float* Linv)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ Flow128 f;
    __shared__ __align__(16) int exps[2][2][C2];          // [buffer][rows, columns] scales
    __shared__ float rmax[2][C2];
    __shared__ int ticket;
    const int nb = cpad128(gs->M) / C2, nbc = mem.rows / C2;
    int* ready = mem.flags;
    int* inv = ready + (size_t)nbc * nbc;
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    if (tid == 0) {
        for (int s = 0; s < C2_STAGES; s++) { mbar_init(&f.full[s], 1); mbar_init(&f.empty[s], 1); }
        for (int b = 0; b < 2; b++) {
            mbar_init(&f.acc_full[b], 1);
            mbar_init(&f.acc_empty[b], C2_EPI);
            mbar_init(&f.exp_full[b], 1);
            mbar_init(&f.sol[b], 1);
        }
        mbar_init(&f.b_full, 1);
        mbar_init(&f.done, 1);
        f.n_issued = f.n_used = f.n_exp = 0;
        f.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&f.tmem)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = f.tmem;

    int it0 = 0, kc0 = 0, nsol = 0;              // stages, column blocks and panel solves so far
    int j = 0, base = 0;                         // the ticket's column; the tickets before that column
    while (true) {
        if (tid == 0) ticket = atomicAdd(inv + nbc, 1);
        __syncthreads();
        const int tk = ticket;
        while (j < nb && tk >= base + min(nb - j, band + 1)) { base += min(nb - j, band + 1); j++; }
        if (j >= nb) break;
        const int i = j + tk - base;
        const bool diag = i == j;
        const int k0 = max(0, i - band), nk = j - k0;
        const int r = 32 * (warp & 3) + lane, h = (warp >> 2) & 1;       // an epilogue thread's row and column half
        const int row = i * C2 + r;
        float acc[64];
        if (warp == C2_EPI) {
            if (lane == 0) {
                bool ok = true;
                for (int k = k0; k < j && ok; k++) {
                    const int kc = kc0 + k - k0, b = kc & 1;
                    const int* rk = ready + (size_t)k * nbc;
                    ok = c2_wait_flag(rk + i, gs, &f.abort) && (diag || c2_wait_flag(rk + j, gs, &f.abort)) &&
                         (kc < 2 || mbar_wait_bounded(&f.acc_empty[b], ((kc >> 1) & 1) ^ 1, &f.abort));
                    if (!ok) break;
                    asm volatile("fence.proxy.async;" ::: "memory");
                    const int* pe = mem.pexp + (size_t)k * mem.rows;
                    mbar_expect_tx(&f.exp_full[b], 2 * C2 * 4);
                    bulk_load(exps[b][0], pe + i * C2, C2 * 4, &f.exp_full[b]);
                    bulk_load(exps[b][1], pe + j * C2, C2 * 4, &f.exp_full[b]);
                    f.n_exp = kc + 1;
                    for (int half = 0; half < 2 && ok; half++) {
                        const int it = it0 + 2 * (k - k0) + half, s = it % C2_STAGES, x = (k % mem.wb) * C2 + half * 64;
                        if (it >= C2_STAGES)
                            ok = mbar_wait_bounded(&f.empty[s], ((it / C2_STAGES) & 1) ^ 1, &f.abort);
                        if (!ok) break;
                        unsigned char* st = smem + s * C2_STAGE_BYTES;
                        mbar_expect_tx(&f.full[s], diag ? 2 * TC_TILE_BYTES : 4 * TC_TILE_BYTES);
                        tma_load_2d(&map_hi, &f.full[s], st, x, i * C2);
                        tma_load_2d(&map_lo, &f.full[s], st + TC_TILE_BYTES, x, i * C2);
                        if (!diag) {
                            tma_load_2d(&map_hi, &f.full[s], st + 2 * TC_TILE_BYTES, x, j * C2);
                            tma_load_2d(&map_lo, &f.full[s], st + 3 * TC_TILE_BYTES, x, j * C2);
                        }
                        f.n_issued = it + 1;
                    }
                }
            }
            __syncwarp();
        } else if (warp == C2_EPI + 1) {
            if (lane == 0) {
                const uint32_t idesc = idesc_f16_128x128();
                int n = 0;
                bool ok = true;
                for (int k = 0; k < nk && ok; k++) {
                    const int kc = kc0 + k, b = kc & 1;
                    ok = kc < 2 || mbar_wait_bounded(&f.acc_empty[b], ((kc >> 1) & 1) ^ 1, &f.abort);
                    for (int half = 0; half < 2 && ok; half++) {
                        const int it = it0 + 2 * k + half, s = it % C2_STAGES;
                        ok = mbar_wait_bounded(&f.full[s], (it / C2_STAGES) & 1, &f.abort);
                        if (!ok) break;
                        tc_fence_after();
                        const uint32_t st = smem_u32(smem + s * C2_STAGE_BYTES);
                        const uint64_t a_hi = sdesc_sw128(st), a_lo = sdesc_sw128(st + TC_TILE_BYTES);
                        const uint64_t b_hi = diag ? a_hi : sdesc_sw128(st + 2 * TC_TILE_BYTES);
                        const uint64_t b_lo = diag ? a_lo : sdesc_sw128(st + 3 * TC_TILE_BYTES);
                        #pragma unroll
                        for (int kk = 0; kk < 4; kk++) {
                            const uint64_t off = (uint64_t)((kk * 32) >> 4);     // 16 F16 = 32 bytes along K
                            mma_f16(tmem + b * C2, a_hi + off, b_hi + off, idesc, (half > 0 || kk > 0) ? 1u : 0u);
                            mma_f16(tmem + b * C2, a_hi + off, b_lo + off, idesc, 1u);
                            mma_f16(tmem + b * C2, a_lo + off, b_hi + off, idesc, 1u);
                        }
                        mma_commit(&f.empty[s]);
                        n = 2 * k + half + 1;
                    }
                    if (ok) mma_commit(&f.acc_full[b]);
                }
                f.n_used = it0 + n;
            }
            __syncwarp();
        } else {
            const float* src = A + (size_t)row * ld + j * C2 + 64 * h;
            #pragma unroll
            for (int c = 0; c < 64; c += 4) {
                const float4 v = *reinterpret_cast<const float4*>(src + c);
                acc[c] = v.x; acc[c + 1] = v.y; acc[c + 2] = v.z; acc[c + 3] = v.w;
            }
            const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(64 * h);
            #pragma unroll 1
            for (int k = 0; k < nk; k++) {
                const int kc = kc0 + k, b = kc & 1;
                if (!mbar_wait_warp(&f.exp_full[b], (kc >> 1) & 1, &f.abort)) break;
                if (!mbar_wait_warp(&f.acc_full[b], (kc >> 1) & 1, &f.abort)) break;
                tc_fence_after();
                const int si = 127 - exps[b][0][r];
                const int* sj = &exps[b][1][64 * h];
                #pragma unroll
                for (int c = 0; c < 64; c += 32) {
                    float v[32];
                    tmem_ld_32cols(trow + (uint32_t)(b * C2 + c), v);
                    #pragma unroll
                    for (int q = 0; q < 32; q += 4) {
                        // 2^-(s_i + s_j), exact (|s_i + s_j| <= 120)
                        const int4 e = *reinterpret_cast<const int4*>(sj + c + q);
                        acc[c + q] -= v[q] * __int_as_float((si - e.x) << 23);
                        acc[c + q + 1] -= v[q + 1] * __int_as_float((si - e.y) << 23);
                        acc[c + q + 2] -= v[q + 2] * __int_as_float((si - e.z) << 23);
                        acc[c + q + 3] -= v[q + 3] * __int_as_float((si - e.w) << 23);
                    }
                }
                tc_fence_before();
                __syncwarp();
                if (lane == 0) c2_arrive(&f.acc_empty[b]);
            }
        }
        it0 += 2 * nk;
        kc0 += nk;
        __syncthreads();                          // every MMA has read its stage: the buffers are free

        if (diag) {
            if (warp < C2_EPI) {
                float* ps = reinterpret_cast<float*>(smem);
                #pragma unroll
                for (int c = 0; c < 64; c++) ps[r * (C2 + 1) + 64 * h + c] = (64 * h + c <= r) ? acc[c] : 0.f;
                c2_sync();
                float* Ajj = A + (size_t)j * C2 * ld + j * C2;
                potrf128(ps, j * C2, which ? &gs->not_spd_R : &gs->not_spd_F,
                         mem.ih + (size_t)j * C2 * C2, mem.il + (size_t)j * C2 * C2);
                asm volatile("fence.proxy.async;" ::: "memory");
                __threadfence();
                c2_sync();
                if (tid == 0) st_release(inv + j, 1);
                potrf128_store(ps, Ajj, ld, Linv ? Linv + (size_t)j * 2 * C2 * C2 : nullptr);
            }
        } else {
            // [quarter 0, 1][A hi, lo] | [quarter 2, 3][A hi, lo] | [two quarters][B hi, lo]
            unsigned char* const at = smem;
            unsigned char* const bt = smem + 8 * TC_TILE_BYTES;
            if (warp == C2_EPI) {
                if (lane == 0 && c2_wait_flag(inv + j, gs, &f.abort)) {
                    asm volatile("fence.proxy.async;" ::: "memory");
                    for (int rd = 0; rd < 2; rd++) {
                        if (rd == 1 && !mbar_wait_bounded(&f.sol[0], nsol & 1, &f.abort)) break;
                        mbar_expect_tx(&f.b_full, 4 * TC_TILE_BYTES);
                        for (int u = 0; u < 2; u++) {
                            tma_load_2d(&map_ih, &f.b_full, bt + (2 * u) * TC_TILE_BYTES, (2 * rd + u) * 32, j * C2);
                            tma_load_2d(&map_il, &f.b_full, bt + (2 * u + 1) * TC_TILE_BYTES, (2 * rd + u) * 32, j * C2);
                        }
                        // landed before the buffers are used again, whatever the others do
                        mbar_wait_bounded(&f.b_full, rd, &f.abort, false);
                    }
                }
                __syncwarp();
            } else if (warp == C2_EPI + 1) {
                asm volatile("bar.sync 2, 288;" ::: "memory");
                if (lane == 0) {
                    const uint32_t idesc = idesc_tf32_128x128(), d = tmem + 2 * C2;
                    for (int rd = 0; rd < 2; rd++) {
                        if (!mbar_wait_bounded(&f.b_full, rd, &f.abort)) break;
                        tc_fence_after();
                        for (int u = 0; u < 2; u++) {
                            const int qt = 2 * rd + u;
                            const uint64_t a_hi = sdesc_sw128(smem_u32(at + (2 * qt) * TC_TILE_BYTES));
                            const uint64_t a_lo = sdesc_sw128(smem_u32(at + (2 * qt + 1) * TC_TILE_BYTES));
                            const uint64_t b_hi = sdesc_sw128(smem_u32(bt + (2 * u) * TC_TILE_BYTES));
                            const uint64_t b_lo = sdesc_sw128(smem_u32(bt + (2 * u + 1) * TC_TILE_BYTES));
                            #pragma unroll
                            for (int kk = 0; kk < TC_KB / 8; kk++) {
                                const uint64_t off = (uint64_t)((kk * 32) >> 4);
                                mma_tf32(d, a_hi + off, b_hi + off, idesc, (qt > 0 || kk > 0) ? 1u : 0u);
                                mma_tf32(d, a_hi + off, b_lo + off, idesc, 1u);
                                mma_tf32(d, a_lo + off, b_hi + off, idesc, 1u);
                            }
                        }
                        mma_commit(&f.sol[rd]);
                    }
                }
                __syncwarp();
            } else {
                #pragma unroll
                for (int c = 0; c < 64; c += 4) {
                    float2 v[4];
                    #pragma unroll
                    for (int e = 0; e < 4; e++) v[e] = split_tf32(acc[c + e]);
                    unsigned char* t = at + (2 * (2 * h + (c >> 5))) * TC_TILE_BYTES + sw128_offset(r, c & 31);
                    *reinterpret_cast<float4*>(t) = make_float4(v[0].x, v[1].x, v[2].x, v[3].x);
                    *reinterpret_cast<float4*>(t + TC_TILE_BYTES) = make_float4(v[0].y, v[1].y, v[2].y, v[3].y);
                }
                asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
                tc_fence_before();
                asm volatile("bar.sync 2, 288;" ::: "memory");
                const bool ok = mbar_wait_warp(&f.sol[1], nsol & 1, &f.abort);
                tc_fence_after();
                const uint32_t trow = tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)(2 * C2 + 64 * h);
                float mx = 0.f;
                if (ok) {
                    #pragma unroll
                    for (int c = 0; c < 64; c += 32) {
                        float v[32];
                        tmem_ld_32cols(trow + (uint32_t)c, v);
                        #pragma unroll
                        for (int q = 0; q < 32; q++) { acc[c + q] = v[q]; mx = fmaxf(mx, fabsf(v[q])); }
                    }
                    tc_fence_before();
                }
                rmax[h][r] = mx;
                c2_sync();
                mx = fmaxf(rmax[0][r], rmax[1][r]);
                int e = 0;
                frexpf(mx, &e);                      // mx < 2^e
                // kept within [-60, 60] so that 2^-(s_i + s_j) is a normal float
                const int sc = (mx > 0.f) ? max(-60, min(60, 14 - e)) : 0;
                if (h == 0) mem.pexp[(size_t)j * mem.rows + row] = sc;
                const float scf = __int_as_float((127 + sc) << 23);
                const size_t at16 = (size_t)row * mem.wb * C2 + (j % mem.wb) * C2 + 64 * h;
                #pragma unroll
                for (int c = 0; c < 64; c += 8) {
                    uint32_t hw[4], lw[4];
                    #pragma unroll
                    for (int q = 0; q < 4; q++) {
                        const float a = acc[c + 2 * q] * scf, b = acc[c + 2 * q + 1] * scf;
                        const __half ah = __float2half_rn(a), bh = __float2half_rn(b);
                        const __half al = __float2half_rn(a - __half2float(ah)), bl = __float2half_rn(b - __half2float(bh));
                        hw[q] = (uint32_t)__half_as_ushort(ah) | ((uint32_t)__half_as_ushort(bh) << 16);
                        lw[q] = (uint32_t)__half_as_ushort(al) | ((uint32_t)__half_as_ushort(bl) << 16);
                    }
                    *reinterpret_cast<uint4*>(mem.Lh + at16 + c) = make_uint4(hw[0], hw[1], hw[2], hw[3]);
                    *reinterpret_cast<uint4*>(mem.Ll + at16 + c) = make_uint4(lw[0], lw[1], lw[2], lw[3]);
                }
                asm volatile("fence.proxy.async;" ::: "memory");
                __threadfence();
                c2_sync();
                if (tid == 0 && !f.abort) st_release(ready + (size_t)j * nbc + i, 1);
                float* dst = A + (size_t)row * ld + j * C2 + 64 * h;
                #pragma unroll
                for (int c = 0; c < 64; c += 4)
                    *reinterpret_cast<float4*>(dst + c) = make_float4(acc[c], acc[c + 1], acc[c + 2], acc[c + 3]);
            }
            nsol++;
        }
        __syncthreads();                          // the one place to leave early: here nobody raises f.abort
        if (f.abort) break;
    }
    if (tid == 32 * (C2_EPI + 1)) mma_commit(&f.done);
    __syncwarp();
    __syncthreads();
    mbar_wait_bounded(&f.done, 0, &f.abort, false);
    if (f.abort && tid == 0)                       // copies issued but never consumed land before the CTA ends
        for (int it = f.n_used; it < f.n_issued; it++)
            mbar_wait_bounded(&f.full[it % C2_STAGES], (it / C2_STAGES) & 1, &f.abort, false);
    if (f.abort && tid == 0)
        for (int kc = max(0, f.n_exp - 2); kc < f.n_exp; kc++)
            mbar_wait_bounded(&f.exp_full[kc & 1], (kc >> 1) & 1, &f.abort, false);
    tc_fence_after();
    tc_fence_before();
    __syncthreads();
    if (f.abort && tid == 0) atomicExch(&gs->status, QLP_ERR_TIMEOUT);
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(512) : "memory");
    }
}

// ---------------------------------------------------------------------------
// F z = r with the factor of k_chol128 and the inverses of
// its 128x128 diagonal blocks (Linv: per block the inverse and its transpose):
//   forward  y_k = Linv_k (r_k - sum_{j<k} L_kj y_j)
//   backward z_k = Linv_k^T (y_k - sum_{j>k} L_jk^T z_j)
// One CTA per block row; CTA k folds in block j as soon as block j's result
// is published (its flag set with release semantics after the values), so
// the long sums spread over many SMs and only the last block of each sum is
// on the critical path.  Every CTA waits only on CTAs with a smaller index,
// which are scheduled before it (the forward-progress assumption of
// single-pass GPU scans), and every wait is bounded by ~1 s of %globaltimer,
// after which the CTA raises QLP_ERR_TIMEOUT and stops.
// ---------------------------------------------------------------------------
// Thread 0 waits until flags[j] is set, then counts how many of the flags
// j .. jend-1 are set in a row; the count (0 on timeout) is broadcast.
__device__ __forceinline__ int wait_ready(const int* flags, int j, int jend, int step, GridState* gs, int* sh)
{
    if (threadIdx.x == 0) {
        int n = 0;
        if (!ld_acquire(flags + j)) {
            const uint64_t t0 = globaltimer();
            while (!ld_acquire(flags + j)) {
                if (*(volatile int*)&gs->status == QLP_ERR_TIMEOUT) break;     // another CTA gave up
                if (globaltimer() - t0 > TC_WAIT_NS) { atomicExch(&gs->status, QLP_ERR_TIMEOUT); break; }
                __nanosleep(64);
            }
        }
        if (ld_acquire(flags + j)) {
            n = 1;
            for (int q = j + step; q != jend && ld_acquire(flags + q); q += step) n++;
        }
        *sh = n;
    }
    __syncthreads();
    const int n = *sh;
    __syncthreads();
    return n;
}

__global__ void __launch_bounds__(256) k_trsv128_fwd(const float* __restrict__ L, int ld,
                                                     const float* __restrict__ Linv, GridState* gs,
                                                     const double* __restrict__ r, float* y, int* flags)
{
    __shared__ float t[C2];
    __shared__ float red[8][C2 / 8];
    __shared__ int sh;
    const int M = gs->M, nb = cpad128(M) / C2;
    const int k = blockIdx.x;
    if (k >= nb) return;
    const int o = k * C2, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // the diagonal block's inverse rows (two threads per row) and, before each
    // wait, this thread's part of the next block of L's strip are loaded
    // first: their latency overlaps the wait for the block they multiply
    const int irow = tid >> 1, ih = tid & 1;
    float4 lv[16];
    {
        const float4* Lr =
            reinterpret_cast<const float4*>(Linv + (size_t)k * 2 * C2 * C2 + (size_t)irow * C2 + ih * 64);
        #pragma unroll
        for (int u = 0; u < 16; u++) lv[u] = Lr[u];
    }
    float part[16];
    #pragma unroll
    for (int i = 0; i < 16; i++) part[i] = 0.f;
    for (int j = 0; j < k;) {
        float4 lp[16];
        #pragma unroll
        for (int i = 0; i < 16; i++)
            lp[i] = *reinterpret_cast<const float4*>(L + (size_t)(o + warp * 16 + i) * ld + j * C2 + 4 * lane);
        const int n = wait_ready(flags, j, k, 1, gs, &sh);
        if (n == 0) return;
        for (int jj = j; jj < j + n; jj++) {
            const float4 yv = __ldcg(reinterpret_cast<const float4*>(y + (size_t)jj * C2) + lane);
            #pragma unroll
            for (int i = 0; i < 16; i++) {
                const float4 lw = (jj == j) ? lp[i]
                    : *reinterpret_cast<const float4*>(L + (size_t)(o + warp * 16 + i) * ld + jj * C2 + 4 * lane);
                part[i] += lw.x * yv.x + lw.y * yv.y + lw.z * yv.z + lw.w * yv.w;
            }
        }
        j += n;
    }
    #pragma unroll
    for (int i = 0; i < 16; i++)
        for (int off = 16; off > 0; off >>= 1) part[i] += __shfl_xor_sync(0xffffffffu, part[i], off);
    if (lane == 0)
        #pragma unroll
        for (int i = 0; i < 16; i++) red[warp][i] = part[i];
    __syncthreads();
    if (tid < C2) t[tid] = ((o + tid < M) ? (float)r[o + tid] : 0.f) - red[tid >> 4][tid & 15];
    __syncthreads();
    {   // y_k = Linv_k t: two threads per row, a half row each
        float acc = 0.f;
        #pragma unroll
        for (int u = 0; u < 16; u++) {
            const int m = ih * 64 + 4 * u;
            acc += lv[u].x * t[m] + lv[u].y * t[m + 1] + lv[u].z * t[m + 2] + lv[u].w * t[m + 3];
        }
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        if (ih == 0) y[o + irow] = acc;
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) st_release(flags + k, 1);
}

__global__ void __launch_bounds__(256) k_trsv128_bwd(const float* __restrict__ L, int ld,
                                                     const float* __restrict__ Linv, GridState* gs,
                                                     const float* __restrict__ y, float* zf,
                                                     double* __restrict__ zout, int* flags)
{
    __shared__ float t[C2];
    __shared__ float red[8][C2];
    __shared__ int sh;
    const int M = gs->M, nb = cpad128(M) / C2;
    const int b = blockIdx.x;
    if (b >= nb) return;
    const int kb = nb - 1 - b, o = kb * C2, tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    // as in the forward sweep: the inverse's rows and, before each wait, the
    // next block of L's column strip are loaded first
    const int ic = tid >> 1, ih = tid & 1;
    float4 lv[16];
    {
        const float4* Lr =
            reinterpret_cast<const float4*>(Linv + (size_t)kb * 2 * C2 * C2 + C2 * C2 + (size_t)ic * C2 + ih * 64);
        #pragma unroll
        for (int u = 0; u < 16; u++) lv[u] = Lr[u];
    }
    float4 part = make_float4(0.f, 0.f, 0.f, 0.f);
    for (int j = nb - 1; j > kb;) {
        float4 lp[16];
        #pragma unroll
        for (int i = 0; i < 16; i++)
            lp[i] = *reinterpret_cast<const float4*>(L + (size_t)(j * C2 + warp * 16 + i) * ld + o + 4 * lane);
        const int n = wait_ready(flags, j, kb, -1, gs, &sh);
        if (n == 0) return;
        for (int jj = j; jj > j - n; jj--) {
            #pragma unroll
            for (int i = 0; i < 16; i++) {
                const int row = jj * C2 + warp * 16 + i;
                const float zv = __ldcg(zf + row);
                const float4 lw = (jj == j) ? lp[i] : *reinterpret_cast<const float4*>(L + (size_t)row * ld + o + 4 * lane);
                part.x += lw.x * zv; part.y += lw.y * zv; part.z += lw.z * zv; part.w += lw.w * zv;
            }
        }
        j -= n;
    }
    red[warp][4 * lane] = part.x; red[warp][4 * lane + 1] = part.y;
    red[warp][4 * lane + 2] = part.z; red[warp][4 * lane + 3] = part.w;
    __syncthreads();
    if (tid < C2) {
        float acc = 0.f;
        #pragma unroll
        for (int w = 0; w < 8; w++) acc += red[w][tid];
        t[tid] = y[o + tid] - acc;
    }
    __syncthreads();
    {   // z_k = Linv_k^T t from the stored transpose: two threads per row of it
        float acc = 0.f;
        #pragma unroll
        for (int u = 0; u < 16; u++) {
            const int m = ih * 64 + 4 * u;
            acc += lv[u].x * t[m] + lv[u].y * t[m + 1] + lv[u].z * t[m + 2] + lv[u].w * t[m + 3];
        }
        acc += __shfl_xor_sync(0xffffffffu, acc, 1);
        if (ih == 0) { zf[o + ic] = acc; zout[o + ic] = (double)acc; }
    }
    __threadfence();
    __syncthreads();
    if (tid == 0) st_release(flags + kb, 1);
}

}  // namespace qlpix
