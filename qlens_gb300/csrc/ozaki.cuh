// ozaki.cuh -- FP64-accurate products A B^T on the tensor cores.
//
// GB300 runs FP64 at 1/64 of FP32 (2 FMA a clock and SM), so an FP64
// contraction is bound by that pipe long before memory or the tensor cores
// matter.  Here a contraction of FP64 operands is split into exact integer
// products (the error-free slicing of Ozaki, Ogita, Oishi & Rump, Numer.
// Algorithms 59, 2012): each row of an operand is scaled by a power of two and
// rounded to 54-bit integers, these are cut into OZ_S = 7 balanced base-256
// digits (-128 .. 127, exact in F16), and the digit products run on tcgen05
// kind::f16.  A product of two digits is at most 2^14, and OZ_FLUSH stages
// (128 terms) of at most 7 digit pairs per weight stay below 2^24, so the FP32
// accumulators hold exact integers; they are then added into 64-bit integers.
// Digit pairs (i, j) with i + j <= 6 are kept (28 of 49): what is left out and
// the rounding of the operands are each ~2^-54 of the rows' largest entries
// per term, with no rounding between terms -- below the rounding error of an
// FP64 sum of the same products.  The sums are integers, so they do not depend
// on how the terms are split over stages, CTAs or launches.
//
// One CTA computes a 128 x 64 tile: warps 0-7 read the accumulators (a warp
// per 32 lanes and 32 columns), warp 8 loads by TMA, warp 9 issues the MMAs.
// The seven weights' accumulators (7 x 64 TMEM columns) form two groups,
// weights 0-3 (10 digit pairs) and 4-6 (18): while the epilogue adds up one
// group, the MMAs of the other run.  Every wait is bounded (~1 s).
#pragma once
#include "tc_common.cuh"

namespace qlpix {

#define OZ_S 7                                   // digits of an operand
#define OZ_TM 128                                // rows of a tile
#define OZ_TN 64                                 // columns of a tile
#define OZ_KS 32                                 // terms per stage (64-byte rows)
#define OZ_FLUSH 4                               // stages between two reads of the accumulators
#define OZ_A_BYTES (OZ_TM * OZ_KS * 2)           // one digit of A: 8 KB
#define OZ_B_BYTES (OZ_TN * OZ_KS * 2)           // ... of B: 4 KB
#define OZ_STAGE_BYTES (OZ_S * (OZ_A_BYTES + OZ_B_BYTES))
#define OZ_STAGES 2
#define OZ_SMEM (OZ_STAGES * OZ_STAGE_BYTES + 1024)
#define OZ_EPI 8                                 // epilogue warps
#define OZ_THREADS (32 * (OZ_EPI + 2))
#define OZ_BITS 54                               // |integer| <= 2^54

struct OzPipe {
    uint64_t full[OZ_STAGES], empty[OZ_STAGES];
    uint64_t acc_full[2], acc_empty[2];          // per accumulator group
    uint64_t done;                               // every MMA issued has completed
    uint32_t tmem;
    int n_issued, n_used;                        // stages loaded / consumed
    volatile int abort;
};

// Shared-memory matrix descriptor: K-major, 64-byte swizzle, 8-row groups 512
// bytes apart.
__device__ __forceinline__ uint64_t sdesc_sw64(uint32_t saddr)
{
    uint64_t d = 0;
    d |= (uint64_t)((saddr & 0x3FFFF) >> 4);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(512 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)4 << 61;                 // SWIZZLE_64B
    return d;
}

// Instruction descriptor: kind::f16, F16 operands, D = F32, K-major, M = 128, N = 64.
__device__ __forceinline__ uint32_t idesc_f16_128x64()
{
    return (1u << 4) | ((uint32_t)(64 >> 3) << 17) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void mbar_arrive(uint64_t* bar)
{
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// Barriers and TMEM (the whole of it: 448 columns are used).  All threads call
// both; they end in a block barrier.
__device__ __forceinline__ void oz_begin(OzPipe& p)
{
    if (threadIdx.x == 0) {
        for (int s = 0; s < OZ_STAGES; s++) { mbar_init(&p.full[s], 1); mbar_init(&p.empty[s], 1); }
        for (int g = 0; g < 2; g++) { mbar_init(&p.acc_full[g], 1); mbar_init(&p.acc_empty[g], OZ_EPI); }
        mbar_init(&p.done, 1);
        p.n_issued = p.n_used = 0;
        p.abort = 0;
        asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
    }
    __syncwarp();
    if (threadIdx.x < 32) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(&p.tmem)),
                     "r"(512)
                     : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
}

// After the last MMA (p.done committed): copies still in flight land, TMEM is freed.
__device__ __forceinline__ void oz_end(OzPipe& p)
{
    __syncthreads();
    mbar_wait_bounded(&p.done, 0, &p.abort, false);
    if (p.abort && threadIdx.x == 0)
        for (int it = p.n_used; it < p.n_issued; it++)
            mbar_wait_bounded(&p.full[it % OZ_STAGES], (it / OZ_STAGES) & 1, &p.abort, false);
    tc_fence_after();
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x < 32) {
        tc_fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(p.tmem), "r"(512) : "memory");
    }
}

// One stage's TMA loads (one thread): the OZ_S digits of 128 rows of A and 64
// rows of B, terms [x, x + OZ_KS).  Digit d's row r sits at row d * ldr + r of
// the maps.  Returns false if the stage's buffer did not come free in time.
__device__ __forceinline__ bool oz_load_stage(OzPipe& p, unsigned char* smem, int it, const CUtensorMap* mapA,
                                              const CUtensorMap* mapB, int ldr, int x, int rowA, int rowB)
{
    const int s = it % OZ_STAGES;
    if (it >= OZ_STAGES && !mbar_wait_bounded(&p.empty[s], ((it / OZ_STAGES) & 1) ^ 1, &p.abort)) return false;
    unsigned char* st = smem + s * OZ_STAGE_BYTES;
    mbar_expect_tx(&p.full[s], OZ_STAGE_BYTES);
    #pragma unroll
    for (int d = 0; d < OZ_S; d++) {
        tma_load_2d(mapA, &p.full[s], st + d * OZ_A_BYTES, x, d * ldr + rowA);
        tma_load_2d(mapB, &p.full[s], st + OZ_S * OZ_A_BYTES + d * OZ_B_BYTES, x, d * ldr + rowB);
    }
    return true;
}

// The MMAs of one accumulator group on one stage: digit pairs (i, j) with
// W0 <= i + j <= W1, the accumulators started anew when `fresh`.
template <int W0, int W1>
__device__ __forceinline__ void oz_mma_group(uint32_t tmem, const unsigned char* st, bool fresh)
{
    const uint32_t idesc = idesc_f16_128x64();
    const uint64_t a0 = sdesc_sw64(smem_u32(st)), b0 = sdesc_sw64(smem_u32(st + OZ_S * OZ_A_BYTES));
    #pragma unroll
    for (int i = 0; i < OZ_S; i++) {
        #pragma unroll
        for (int kk = 0; kk < 2; kk++) {
            #pragma unroll
            for (int j = 0; j < OZ_S; j++) {
                if (i + j < W0 || i + j > W1) continue;
                const uint64_t a = a0 + (uint64_t)((i * OZ_A_BYTES + kk * 32) >> 4);
                const uint64_t b = b0 + (uint64_t)((j * OZ_B_BYTES + kk * 32) >> 4);
                mma_f16(tmem + (uint32_t)((i + j) * OZ_TN), a, b, idesc, (fresh && i == 0 && kk == 0) ? 0u : 1u);
            }
        }
    }
}

// The MMA issuer (one thread): n stages, the accumulators handed to the
// epilogue every OZ_FLUSH stages.  In a group, weight w's first product is the
// pair (0, w), so it is the one that starts the accumulator.
__device__ __forceinline__ void oz_mma_loop(OzPipe& p, const unsigned char* smem, int n)
{
    int it = 0;
    for (; it < n; it++) {
        const int s = it % OZ_STAGES, fb = it / OZ_FLUSH;
        const bool fresh = it % OZ_FLUSH == 0, last = it % OZ_FLUSH == OZ_FLUSH - 1 || it == n - 1;
        if (!mbar_wait_bounded(&p.full[s], (it / OZ_STAGES) & 1, &p.abort)) break;
        if (fresh && fb > 0 && !mbar_wait_bounded(&p.acc_empty[0], (fb - 1) & 1, &p.abort)) break;
        tc_fence_after();
        const unsigned char* st = smem + s * OZ_STAGE_BYTES;
        oz_mma_group<0, 3>(p.tmem, st, fresh);
        if (last) mma_commit(&p.acc_full[0]);
        if (fresh && fb > 0 && !mbar_wait_bounded(&p.acc_empty[1], (fb - 1) & 1, &p.abort)) break;
        tc_fence_after();
        oz_mma_group<4, 6>(p.tmem, st, fresh);
        mma_commit(&p.empty[s]);
        if (last) mma_commit(&p.acc_full[1]);
    }
    p.n_used = it;
    mma_commit(&p.done);
}

// 16 TMEM columns of the warp's 32 lanes.
__device__ __forceinline__ void tmem_ld_16cols(uint32_t taddr, float (&v)[16])
{
    uint32_t r[16];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 "
        "{%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr));
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
    #pragma unroll
    for (int i = 0; i < 16; i++) v[i] = __uint_as_float(r[i]);
}

// The epilogue warps: the accumulators of n stages added into this thread's
// integers -- row 32 (warp % 4) + lane of the tile, columns 32 (warp / 4) .. + 31.
// The sum of the products is (hi 2^24 + lo) 2^(Ea + Eb - 60) for rows scaled by
// 2^(54 - Ea), 2^(54 - Eb); lo stays in [0, 2^24), its carry goes to hi, so
// that the 32 columns' sums and a load fit the 168 registers that ten warps
// leave a thread.
__device__ __forceinline__ bool oz_accumulate(OzPipe& p, int n, long long (&hi)[32], int (&lo)[32])
{
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = p.tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * 32);
    const int nf = (n + OZ_FLUSH - 1) / OZ_FLUSH;
    #pragma unroll 1
    for (int fb = 0; fb < nf; fb++) {
        float v[16];
        if (!mbar_wait_bounded(&p.acc_full[0], fb & 1, &p.abort)) return false;
        tc_fence_after();
        #pragma unroll
        for (int h = 0; h < 32; h += 16) {
            #pragma unroll
            for (int w = 0; w < 4; w++) {
                tmem_ld_16cols(base + (uint32_t)(w * OZ_TN + h), v);
                #pragma unroll
                for (int c = 0; c < 16; c++)
                    hi[h + c] += (long long)__float2int_rn(v[c]) * (long long)(1 << (8 * (3 - w)));
            }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p.acc_empty[0]);
        if (!mbar_wait_bounded(&p.acc_full[1], fb & 1, &p.abort)) return false;
        tc_fence_after();
        #pragma unroll
        for (int h = 0; h < 32; h += 16) {
            long long t[16];
            #pragma unroll
            for (int w = 4; w < 7; w++) {
                tmem_ld_16cols(base + (uint32_t)(w * OZ_TN + h), v);
                #pragma unroll
                for (int c = 0; c < 16; c++)
                    t[c] = (w == 4 ? (long long)lo[h + c] : t[c]) +
                           (long long)__float2int_rn(v[c]) * (long long)(1 << (8 * (6 - w)));
            }
            #pragma unroll
            for (int c = 0; c < 16; c++) {
                hi[h + c] += t[c] >> 24;
                lo[h + c] = (int)t[c] & 0xffffff;
            }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p.acc_empty[1]);
    }
    return true;
}

// The biased exponent of |x| (at least 1), 0 for zero, 2047 for infinities and NaN.
__device__ __forceinline__ int oz_exponent(double x)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(x) << 1;
    return u == 0 ? 0 : max(1, (int)(u >> 53));
}

// x as an integer on the grid of a row whose largest biased exponent is emax:
// round(x 2^(54 - E)), E = emax - 1022 (|x| < 2^E); integer arithmetic only.
// Past the range (a row's bound that does not hold) it saturates.
__device__ __forceinline__ long long oz_fixed(double x, int emax)
{
    const long long b = __double_as_longlong(x);
    int e = (int)((b >> 52) & 0x7ff);
    long long m = b & 0xfffffffffffffll;
    if (e > 0) m |= 1ll << 52; else e = 1;
    const int sh = emax - e;                        // q = m 2^(1 - sh)
    long long q;
    if (sh <= 0) q = sh == 0 ? (m << 1) : (m ? (1ll << OZ_BITS) : 0);
    else if (sh == 1) q = m;
    else if (sh < 56) q = (m + (1ll << (sh - 2))) >> (sh - 1);
    else q = 0;
    return b < 0 ? -q : q;
}

// 2^(emax - 1022): what a unit of 2^54 of the grid stands for; NaN for a row
// that holds an infinity or a NaN.
__device__ __forceinline__ double oz_scale(int emax)
{
    if (emax >= 2047) return __longlong_as_double(0x7ff8000000000000ll);
    // 2^(emax - 1022) = 2 * 2^(emax - 1023), the inner factor formed by its bits
    return emax <= 0 ? 0.0 : 2.0 * __longlong_as_double((long long)emax << 52);
}

// Two integers' digits of weight 256^(6 - d) as a pair of F16 (a low half).
// Each integer carries the bias 0x0080808080808080 (added once by oz_bias), so
// that its bytes are digit + 128; the top digit keeps its sign.
__device__ __forceinline__ unsigned long long oz_bias(long long q)
{
    return (unsigned long long)(q + 0x0080808080808080ll);
}

__device__ __forceinline__ uint32_t oz_digits(unsigned long long qa, unsigned long long qb, int d)
{
    // byte b of F16 pattern 0x6400 | b is 1024 + b
    const int sh = 8 * (6 - d);
    const uint32_t a = (uint32_t)(qa >> sh) & 0xffu, b = (uint32_t)(qb >> sh) & 0xffu;
    uint32_t h = 0x64006400u | a | (b << 16);
    uint32_t r;
    // 1024 + 128 = 1152 = 0x6480
    asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r) : "r"(h), "r"(0x64806480u));
    return r;
}

}  // namespace qlpix
