// tc_syrk.cuh -- F = X X^T on the 5th-generation tensor cores (tcgen05).
//
// X is L'^T scaled by sqrt(C^-1): M_cap rows (source cells) x K_cap columns
// (image pixels), K contiguous, split into a rounded high part and a rounded
// remainder so that hi*hi + hi*lo + lo*hi carries ~22 bits.  The parts are F16
// (kind::f16, K = 16 per MMA, 64 pixels per 128-byte stage row): as many
// significant bits as TF32 at twice the tensor rate, X scaled by a power of two so
// that its largest entry is near 2^14, undone exactly in the epilogue.  One CTA
// computes one 128x128 tile of the lower triangle of F:
//   warp 0 / lane 0  TMA producer: 128-row boxes of 128 B (128 B swizzle) of
//                    X_hi, X_lo for the tile's row block and column block
//                    into a 3-stage shared-memory ring;
//   warp 1 / lane 0  MMA issuer, 4 k-steps of tcgen05.mma.cta_group::1 per stage
//                    into FP32 accumulators in TMEM: hi*(hi, lo) as one
//                    N = 256 product (lo's rows follow hi's in shared memory) and
//                    lo*hi into the second half;
//   all 4 warps      epilogue: tcgen05.ld 32x32b.x32, the halves added, FP32
//                    stores to F.
// Block sparsity: a stage is processed only if both the row block and the
// column block of X have a nonzero among its pixels (flags per 32 pixels from
// the PSF-to-X build), so the work follows the overlap of the two source-cell
// blocks' footprints in the image instead of the full pixel count.
// All threads list the live stages before the first is loaded.
// What bounds it: shared memory (an N = 128 product of F16 reads its 128 bytes a
// clock, the N = 256 one less) and L2, which feeds a CTA 64 KB per 768 clocks of
// products; the tensor pipe ran at 40 %.  Two single threads that tested every
// stage as they came to it lost the time of the dead ones.  us, three products and
// tests as they came -> now: 2,934 cells x 11,772 pixels 130 -> 95, 3,700 x 42,700
// 262 -> 186, 2,304 x 40,000 292 -> 241, 738 x 6,220 51 -> 40.
// Every mbarrier wait is bounded by ~1 s of %globaltimer; on expiry the
// kernel raises QLP_ERR_TIMEOUT in the GridState, stops issuing work, frees
// its TMEM and returns.
#pragma once
#include "tc_common.cuh"

namespace qlpix {

#define TC_LIST 4096              // stages looked through at a time

// grid: one CTA per lower-triangle 128x128 tile of the M_cap x M_cap output.
// nzflags[rb * nkb_cap + kb] != 0 when rows [128 rb, 128 rb + 128) of X have a
// nonzero in columns [32 kb, 32 kb + 32) (a stage's 64 pixels: flags 2 kb and
// 2 kb + 1); fscale multiplies the result (2^-2s for X scaled by 2^s).
__global__ void __launch_bounds__(128, 1) k_syrk_tc(const __grid_constant__ CUtensorMap map_hi,
                                                    const __grid_constant__ CUtensorMap map_lo,
                                                    GridState* gs, const unsigned char* __restrict__ nzflags,
                                                    int nkb_cap, float* __restrict__ F, int ldF, float fscale)
{
    constexpr int KPS = 2 * TC_KB;                     // pixels per stage (128 bytes of a row)
    extern __shared__ unsigned char smem_raw[];
    __shared__ uint64_t full_bar[TC_STAGES];
    __shared__ uint64_t empty_bar[TC_STAGES];
    __shared__ uint64_t done_bar;
    __shared__ uint32_t tmem_slot;
    __shared__ int n_active;
    __shared__ int n_issued;
    __shared__ int wsum[4];
    __shared__ unsigned short live_kb[TC_LIST];
    __shared__ volatile int abort_flag;

    int bi, bj;
    {
        int t = blockIdx.x;
        int i = (int)((sqrt(8.0 * t + 1.0) - 1.0) * 0.5);
        while ((i + 1) * (i + 2) / 2 <= t) i++;
        while (i * (i + 1) / 2 > t) i--;
        bi = i;
        bj = t - i * (i + 1) / 2;
    }
    const int M = gs->M, N = gs->N;
    const int Mp = (M + TC_TILE - 1) / TC_TILE * TC_TILE;
    if (bi * TC_TILE >= Mp) return;
    const int nkb = (N + KPS - 1) / KPS;

    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);

    if (threadIdx.x == 0) {
        for (int s = 0; s < TC_STAGES; s++) {
            mbar_init(&full_bar[s], 1);
            mbar_init(&empty_bar[s], 1);
        }
        mbar_init(&done_bar, 1);
        n_active = 0;
        n_issued = 0;
        abort_flag = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (warp == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&tmem_slot)),
                     "r"(2 * TC_TILE)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t tmem = tmem_slot;

    const unsigned char* fi = nzflags + (size_t)bi * nkb_cap;
    const unsigned char* fj = nzflags + (size_t)bj * nkb_cap;
    // stage kb has work when both blocks have a nonzero among its pixels
    auto live = [&](int kb) -> bool {
        return (fi[2 * kb] | fi[2 * kb + 1]) && (fj[2 * kb] | fj[2 * kb + 1]);
    };

    int it_p = 0, it_m = 0;                            // stages loaded (warp 0), multiplied (warp 1)
    for (int k0 = 0; k0 < nkb; k0 += TC_LIST) {
        // ---- the live stages of this stretch, in order, by all threads ----
        const int k1 = min(k0 + TC_LIST, nkb);
        int n = 0;
        for (int c = k0; c < k1; c += 128) {
            const int kb = c + threadIdx.x;
            const bool on = kb < k1 && live(kb);
            const unsigned bits = __ballot_sync(0xffffffffu, on);
            if (lane == 0) wsum[warp] = __popc(bits);
            __syncthreads();
            int at = n + __popc(bits & ((1u << lane) - 1));
            for (int w = 0; w < 4; w++) {
                if (w < warp) at += wsum[w];
                n += wsum[w];
            }
            if (on) live_kb[at] = (unsigned short)(kb - k0);
            __syncthreads();
        }
        if (warp == 0 && lane == 0) {
            // ---- TMA producer ----
            for (int u = 0; u < n; u++, it_p++) {
                const int x = (k0 + live_kb[u]) * KPS, s = it_p % TC_STAGES;
                if (it_p >= TC_STAGES) {
                    if (!mbar_wait_bounded(&empty_bar[s], ((it_p / TC_STAGES) & 1) ^ 1, &abort_flag)) break;
                }
                unsigned char* st = smem + s * TC_STAGE_BYTES;
                mbar_expect_tx(&full_bar[s], TC_STAGE_BYTES);
                tma_load_2d(&map_hi, &full_bar[s], st, x, bi * TC_TILE);
                tma_load_2d(&map_lo, &full_bar[s], st + TC_TILE_BYTES, x, bi * TC_TILE);
                tma_load_2d(&map_hi, &full_bar[s], st + 2 * TC_TILE_BYTES, x, bj * TC_TILE);
                tma_load_2d(&map_lo, &full_bar[s], st + 3 * TC_TILE_BYTES, x, bj * TC_TILE);
            }
            n_issued = it_p;
        } else if (warp == 1 && lane == 0) {
            // ---- MMA issuer ----
            const uint32_t idesc = idesc_f16_128x128();
            const uint32_t idesc2 = idesc_f16(128, 256);
            for (int u = 0; u < n; u++, it_m++) {
                const int s = it_m % TC_STAGES;
                if (!mbar_wait_bounded(&full_bar[s], (it_m / TC_STAGES) & 1, &abort_flag)) break;
                tc_fence_after();
                unsigned char* st = smem + s * TC_STAGE_BYTES;
                const uint64_t a_hi = sdesc_sw128(smem_u32(st));
                const uint64_t a_lo = sdesc_sw128(smem_u32(st + TC_TILE_BYTES));
                const uint64_t b_hi = sdesc_sw128(smem_u32(st + 2 * TC_TILE_BYTES));
                #pragma unroll
                for (int kk = 0; kk < 4; kk++) {
                    // one MMA takes 32 bytes along K: 16 F16 values
                    const uint64_t off = (uint64_t)((kk * 32) >> 4);
                    const uint32_t acc = (it_m > 0 || kk > 0) ? 1u : 0u;
                    // B's lo rows follow its hi rows: hi*hi and hi*lo are one N = 256
                    // product, side by side in TMEM; lo*hi joins hi*lo
                    mma_f16(tmem, a_hi + off, b_hi + off, idesc2, acc);
                    mma_f16(tmem + TC_TILE, a_lo + off, b_hi + off, idesc, 1u);
                }
                mma_commit(&empty_bar[s]);
            }
            n_active = it_m;
        }
        __syncthreads();
        if (abort_flag) break;                         // uniform: raised between the barriers only
    }
    if (warp == 1 && lane == 0) mma_commit(&done_bar);
    __syncthreads();
    // ---- epilogue ----
    // Wait for the committed MMAs even after an abort: TMEM is freed below.
    bool ok = mbar_wait_bounded(&done_bar, 0, &abort_flag, false);
    if (abort_flag && threadIdx.x == 0) {
        // let TMA copies that were issued but never consumed land before exit
        for (int it = n_active; it < n_issued; it++)
            mbar_wait_bounded(&full_bar[it % TC_STAGES], (it / TC_STAGES) & 1, &abort_flag, false);
    }
    ok = __syncthreads_and(ok && !abort_flag);         // the warps' TMEM loads need all their lanes
    tc_fence_after();
    const int row = bi * TC_TILE + warp * 32 + lane;
    float* out = F + (size_t)row * ldF + bj * TC_TILE;
    if (ok && n_active > 0) {
        #pragma unroll 1
        for (int c = 0; c < TC_TILE; c += 32) {
            float v[32];
            const uint32_t taddr = tmem + ((uint32_t)(warp * 32) << 16) + (uint32_t)c;
            tmem_ld_32cols(taddr, v);
            float lo[32];
            tmem_ld_32cols(taddr + TC_TILE, lo);
            #pragma unroll
            for (int i = 0; i < 32; i++) v[i] += lo[i];
            #pragma unroll
            for (int i = 0; i < 32; i += 4)
                *reinterpret_cast<float4*>(out + c + i) =
                    make_float4(v[i] * fscale, v[i + 1] * fscale, v[i + 2] * fscale, v[i + 3] * fscale);
        }
    } else {
        for (int c = 0; c < TC_TILE; c += 4) *reinterpret_cast<float4*>(out + c) = make_float4(0.f, 0.f, 0.f, 0.f);
    }
    tc_fence_before();
    __syncthreads();
    if (abort_flag && threadIdx.x == 0) atomicExch(&gs->status, QLP_ERR_TIMEOUT);
    if (warp == 0) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(2 * TC_TILE) : "memory");
    }
}

}  // namespace qlpix
