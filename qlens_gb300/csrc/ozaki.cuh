// ozaki.cuh -- FP64-accurate products A B^T on the tensor cores.
//
// GB300 runs FP64 at 1/64 of FP32 (2 FMA a clock and SM), so an FP64
// contraction is bound by that pipe long before memory or the tensor cores
// matter.  Here a contraction of FP64 operands is split into exact integer
// products (the error-free slicing of Ozaki, Ogita, Oishi & Rump, Numer.
// Algorithms 59, 2012): each row of an operand is scaled by a power of two and
// rounded to integers of 8 S - 2 bits, these are cut into S balanced base-256
// digits (-128 .. 127, exact in F16), and the digit products run on tcgen05
// kind::f16.  A product of two digits is at most 2^14, and OZ_FLUSH stages
// (128 terms) of at most S <= 8 digit pairs per weight stay within 2^24, so the
// FP32 accumulators hold exact integers; they are then added into wider
// integers.  Digit pairs (i, j) with i + j < S are kept (S = 7: 28 of 49): what
// is left out and the rounding of the operands are each ~2^-(8 S - 2) of the
// rows' largest entries per term, with no rounding between terms.  The sums are
// integers, so they do not depend on how the terms are split over stages, CTAs
// or launches.  S = 7 (54 bits) serves L'^T C^-1 L', whose rows' sums of squares
// are the result's scale; the factorisation takes S = 8 (62 bits): its rows are
// scaled by their norm, well above most of their entries, and with S = 7 log
// det R and the amplitudes came out 3 to 30 times further off than in FP64.
//
// One CTA computes a 128 x 64 tile: warps 0-7 read the accumulators (a warp
// per 32 lanes and 32 columns), warp 8 loads by TMA, warp 9 issues the MMAs.
// The weights' accumulators (S x 64 TMEM columns) form two groups, weights 0-3
// and 4 on: while the epilogue adds up one group, the MMAs of the other run.
// Every wait is bounded (~1 s).
#pragma once
#include "tc_common.cuh"

namespace qlpix {

#define OZ_TM 128                                // rows of a tile
#define OZ_TN 64                                 // columns of a tile
#define OZ_KS 32                                 // terms per stage (64-byte rows)
#define OZ_FLUSH 4                               // stages between two reads of the accumulators
#define OZ_A_BYTES (OZ_TM * OZ_KS * 2)           // one digit of A: 8 KB
#define OZ_B_BYTES (OZ_TN * OZ_KS * 2)           // ... of B: 4 KB
#define OZ_STAGES 2
#define OZ_EPI 8                                 // epilogue warps
#define OZ_THREADS (32 * (OZ_EPI + 2))

__host__ __device__ constexpr int oz_stage_bytes(int S) { return S * (OZ_A_BYTES + OZ_B_BYTES); }
__host__ __device__ constexpr int oz_smem(int S) { return OZ_STAGES * oz_stage_bytes(S) + 1024; }
__host__ __device__ constexpr int oz_bits(int S) { return 8 * S - 2; }      // |integer| <= 2^oz_bits

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

// Barriers and TMEM (the whole of it: 448 or 512 columns are used).  All threads call
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

// One stage's TMA loads (one thread): the S digits of 128 rows of A and 64
// rows of B, terms [x, x + OZ_KS).  Digit d's row r sits at row d * ldr + r of
// the maps.  Returns false if the stage's buffer did not come free in time.
template <int S>
__device__ __forceinline__ bool oz_load_stage(OzPipe& p, unsigned char* smem, int it, const CUtensorMap* mapA,
                                              const CUtensorMap* mapB, int ldr, int x, int rowA, int rowB)
{
    const int s = it % OZ_STAGES;
    if (it >= OZ_STAGES && !mbar_wait_bounded(&p.empty[s], ((it / OZ_STAGES) & 1) ^ 1, &p.abort)) return false;
    unsigned char* st = smem + s * oz_stage_bytes(S);
    mbar_expect_tx(&p.full[s], oz_stage_bytes(S));
    #pragma unroll
    for (int d = 0; d < S; d++) {
        tma_load_2d(mapA, &p.full[s], st + d * OZ_A_BYTES, x, d * ldr + rowA);
        tma_load_2d(mapB, &p.full[s], st + S * OZ_A_BYTES + d * OZ_B_BYTES, x, d * ldr + rowB);
    }
    return true;
}

// An MMA that loads its A rows into the unit's collector for the next ones, and
// one that takes them from there (an N = 64 MMA is otherwise bound by reading A
// from shared memory: 6 KB against 32 clocks of arithmetic).
#define OZ_MMA(NAME, USE)                                                                                             \
    __device__ __forceinline__ void NAME(uint32_t tmem_d, uint64_t adesc, uint64_t bdesc, uint32_t idesc, uint32_t acc) \
    {                                                                                                                \
        asm volatile(                                                                                                \
            "{\n\t.reg .pred p;\n\t"                                                                                 \
            "setp.ne.b32 p, %4, 0;\n\t"                                                                              \
            "tcgen05.mma.cta_group::1.kind::f16.collector::a::" USE " [%0], %1, %2, %3, p;\n\t}" ::"r"(tmem_d),         \
            "l"(adesc), "l"(bdesc), "r"(idesc), "r"(acc)                                                             \
            : "memory");                                                                                             \
    }
OZ_MMA(oz_mma_fill, "fill")
OZ_MMA(oz_mma_use, "use")
OZ_MMA(oz_mma_last, "lastuse")

// The MMAs of one accumulator group on one stage: digit pairs (i, j) with
// W0 <= i + j <= W1, the accumulators started anew when `fresh`.
template <int S, int W0, int W1>
__device__ __forceinline__ void oz_mma_group(uint32_t tmem, const unsigned char* st, bool fresh)
{
    const uint32_t idesc = idesc_f16_128x64();
    const uint64_t a0 = sdesc_sw64(smem_u32(st)), b0 = sdesc_sw64(smem_u32(st + S * OZ_A_BYTES));
    #pragma unroll
    for (int i = 0; i < S; i++) {
        #pragma unroll
        for (int kk = 0; kk < 2; kk++) {
            #pragma unroll
            for (int j = 0; j < S; j++) {
                if (i + j < W0 || i + j > W1) continue;
                const uint64_t a = a0 + (uint64_t)((i * OZ_A_BYTES + kk * 32) >> 4);
                const uint64_t b = b0 + (uint64_t)((j * OZ_B_BYTES + kk * 32) >> 4);
                const uint32_t d = tmem + (uint32_t)((i + j) * OZ_TN), acc = (fresh && i == 0 && kk == 0) ? 0u : 1u;
                const bool first = j == 0 || i + j == W0, last = i + j == W1;
                if (first && last) mma_f16(d, a, b, idesc, acc);
                else if (first) oz_mma_fill(d, a, b, idesc, acc);
                else if (last) oz_mma_last(d, a, b, idesc, acc);
                else oz_mma_use(d, a, b, idesc, acc);
            }
        }
    }
}

// The MMA issuer (one thread): n stages, the accumulators handed to the
// epilogue every OZ_FLUSH stages.  it0, f0: the stages and readings of the
// accumulators that went before (the barriers' phases).  In a group, weight w's
// first product is the pair (0, w), so it is the one that starts the accumulator.
template <int S>
__device__ __forceinline__ void oz_mma_loop(OzPipe& p, const unsigned char* smem, int it0, int f0, int n)
{
    int i = 0;
    for (; i < n; i++) {
        const int it = it0 + i, s = it % OZ_STAGES, f = f0 + i / OZ_FLUSH;
        const bool fresh = i % OZ_FLUSH == 0, last = i % OZ_FLUSH == OZ_FLUSH - 1 || i == n - 1;
        if (!mbar_wait_bounded(&p.full[s], (it / OZ_STAGES) & 1, &p.abort)) break;
        if (fresh && f > 0 && !mbar_wait_bounded(&p.acc_empty[0], (f - 1) & 1, &p.abort)) break;
        tc_fence_after();
        const unsigned char* st = smem + s * oz_stage_bytes(S);
        oz_mma_group<S, 0, 3>(p.tmem, st, fresh);
        if (last) mma_commit(&p.acc_full[0]);
        if (fresh && f > 0 && !mbar_wait_bounded(&p.acc_empty[1], (f - 1) & 1, &p.abort)) break;
        tc_fence_after();
        oz_mma_group<S, 4, S - 1>(p.tmem, st, fresh);
        mma_commit(&p.empty[s]);
        if (last) mma_commit(&p.acc_full[1]);
    }
    p.n_used = it0 + i;
}

// The same for two stage buffers that the CTA's threads filled themselves (64
// terms, reading f of the accumulators).
template <int S>
__device__ __forceinline__ void oz_mma_filled(OzPipe& p, const unsigned char* smem, int f)
{
    if (f > 0 && !mbar_wait_bounded(&p.acc_empty[0], (f - 1) & 1, &p.abort)) return;
    if (f > 0 && !mbar_wait_bounded(&p.acc_empty[1], (f - 1) & 1, &p.abort)) return;
    tc_fence_after();
    oz_mma_group<S, 0, 3>(p.tmem, smem, true);
    oz_mma_group<S, 0, 3>(p.tmem, smem + oz_stage_bytes(S), false);
    mma_commit(&p.acc_full[0]);
    oz_mma_group<S, 4, S - 1>(p.tmem, smem, true);
    oz_mma_group<S, 4, S - 1>(p.tmem, smem + oz_stage_bytes(S), false);
    mma_commit(&p.acc_full[1]);
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

// The epilogue warps: the accumulators of n stages (readings f0, f0 + 1, ...)
// added into this thread's integers -- row 32 (warp % 4) + lane of the tile,
// columns 32 (warp / 4) .. + 31.  With h = 8 (S - 4) the sum of the products is
// (hi 2^h + lo) 2^(Ea + Eb - oz_unit(S)) for rows scaled by 2^(oz_bits(S) - E); lo
// stays in [0, 2^h), its carry goes to hi, so that the 32 columns' sums and a
// load fit the 168 registers that ten warps leave a thread.
__host__ __device__ constexpr int oz_unit(int S) { return 2 * oz_bits(S) - 8 * (S - 1); }

template <int S>
__device__ __forceinline__ bool oz_accumulate(OzPipe& p, int f0, int n, long long (&hi)[32], uint32_t (&lo)[32])
{
    constexpr int H = 8 * (S - 4);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const uint32_t base = p.tmem + ((uint32_t)((warp & 3) * 32) << 16) + (uint32_t)((warp >> 2) * 32);
    const int nf = (n + OZ_FLUSH - 1) / OZ_FLUSH;
    #pragma unroll 1
    for (int f = f0; f < f0 + nf; f++) {
        float v[16];
        if (!mbar_wait_warp(&p.acc_full[0], f & 1, &p.abort)) return false;
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
        if (!mbar_wait_warp(&p.acc_full[1], f & 1, &p.abort)) return false;
        tc_fence_after();
        #pragma unroll
        for (int h = 0; h < 32; h += 16) {
            long long t[16];
            #pragma unroll
            for (int w = 4; w < S; w++) {
                tmem_ld_16cols(base + (uint32_t)(w * OZ_TN + h), v);
                #pragma unroll
                for (int c = 0; c < 16; c++)
                    t[c] = (w == 4 ? (long long)lo[h + c] : t[c]) +
                           (long long)__float2int_rn(v[c]) * (long long)(1 << (8 * (S - 1 - w)));
            }
            #pragma unroll
            for (int c = 0; c < 16; c++) {
                hi[h + c] += t[c] >> H;
                lo[h + c] = H == 32 ? (uint32_t)t[c] : (uint32_t)t[c] & ((1u << (H & 31)) - 1);
            }
        }
        tc_fence_before();
        __syncwarp();
        if (lane == 0) mbar_arrive(&p.acc_empty[1]);
    }
    return true;
}

// Byte offset of the 16-byte chunk that holds terms [8 q, 8 q + 8) of a row in a
// 64-byte-swizzled digit block.
__device__ __forceinline__ uint32_t oz_chunk(int row, int q)
{
    return (uint32_t)(row * 64 + ((q ^ ((row >> 1) & 3)) << 4));
}

// The biased exponent of |x| (at least 1), 0 for zero, 2047 for infinities and NaN.
__device__ __forceinline__ int oz_exponent(double x)
{
    const unsigned long long u = (unsigned long long)__double_as_longlong(x) << 1;
    return u == 0 ? 0 : max(1, (int)(u >> 53));
}

// x as an integer of up to 54 bits (S = 7) on the grid of a row whose largest
// biased exponent is emax: round(x 2^(54 - E)), E = emax - 1022 (|x| < 2^E);
// integer arithmetic only.
__device__ __forceinline__ long long oz_fixed54(double x, int emax)
{
    const long long b = __double_as_longlong(x);
    int e = (int)((b >> 52) & 0x7ff);
    long long m = b & 0xfffffffffffffll;
    if (e > 0) m |= 1ll << 52; else e = 1;
    const int sh = emax - e;                        // q = m 2^(1 - sh)
    long long q;
    if (sh <= 0) q = m << 1;
    else if (sh == 1) q = m;
    else if (sh < 56) q = (m + (1ll << (sh - 2))) >> (sh - 1);
    else q = 0;
    return b < 0 ? -q : q;
}

// 2^(emax - 1022): what 2^54 of the grid stands for; NaN for a row
// that holds an infinity or a NaN.
__device__ __forceinline__ double oz_scale(int emax)
{
    if (emax >= 2047) return __longlong_as_double(0x7ff8000000000000ll);
    // 2^(emax - 1022) = 2 * 2^(emax - 1023), the inner factor formed by its bits
    return emax <= 0 ? 0.0 : 2.0 * __longlong_as_double((long long)emax << 52);
}

// Digits: each integer carries a bias of 128 in every byte (added once by
// oz_bias), so that its bytes are digit + 128; digit d has weight 256^(S-1-d).
template <int S>
__device__ __forceinline__ unsigned long long oz_bias(long long q)
{
    return (unsigned long long)q + (0x8080808080808080ull >> (64 - 8 * S));
}

// Digit d of eight integers as F16: byte b of the pattern 0x6400 | b is 1024 + b,
// and 1024 + 128 = 0x6480 goes off.  Three instructions a pair.
template <int S>
__device__ __forceinline__ uint4 oz_digits8(const unsigned long long* q, int d)
{
    const int k = S - 1 - d;                        // byte
    uint32_t r[4];
    #pragma unroll
    for (int u = 0; u < 4; u++) {
        const uint32_t a = (uint32_t)(k < 4 ? q[2 * u] : q[2 * u] >> 32);
        const uint32_t b = (uint32_t)(k < 4 ? q[2 * u + 1] : q[2 * u + 1] >> 32);
        const uint32_t h = (__byte_perm(a, b, (k & 3) | ((4 + (k & 3)) << 8)) & 0x00ff00ffu) | 0x64006400u;
        asm("sub.rn.f16x2 %0, %1, %2;" : "=r"(r[u]) : "r"(h), "r"(0x64806480u));
    }
    return make_uint4(r[0], r[1], r[2], r[3]);
}

}  // namespace qlpix
