// cholfp64.cu -- the plain path's dense factorisation and solve:
//   F = L L^T and R = L L^T   k_chol64 (one launch each)
//   F again, in FP64          k_chol64_plain, where k_chol64 met a pivot <= 0
//   F s = D                   k_trsv64_fwd, k_trsv64_bwd
// Reference: Cholesky_dcmp_packed (pixelgrid.cpp:17071-17105; a negative pivot
// is flagged and sqrt(|d|) used), Cholesky_solve_lower_packed (17230-17246).
//
// The factorisation is left-looking over 64-column blocks and runs as one grid
// of CTAs that take tiles (128 rows x 64 columns, column by column) from a
// counter.  A tile sums L_ik L_jk^T over the finished columns k < j by digit
// products on the tensor cores (ozaki.cuh), waiting per column block for the
// flags of the rows that it reads; its diagonal 64x64 block is then factored
// and inverted by the CTA itself, and the rows below it become L by a product
// with that inverse, again as digits.  A tile waits only on tiles with a
// smaller number, which are finished or held by running CTAs, so the grid may
// have any size; every wait is bounded (~1 s).
//
// Numbers: row i is scaled by 2^-E_i with E_i = ceil(log2 sqrt(F_ii)), so that
// every entry of the factor and of the Schur complements is at most 1.  Both
// are kept as 64-bit integers, the factor on the grid 2^-62 (eight digits), the
// Schur complements on 2^-60, and the diagonal blocks are factored and inverted
// in integers too: GB300's integer pipes multiply 64-bit numbers several times
// faster than its FP64 pipe (2 FMA a clock and SM), whose latencies had made a
// pivot cost 1.2 us.  An FP64 factorisation rounds at 2^-53 of the same scale per
// operation; log det F, log det R and the amplitudes come out as close to an
// extended-precision factorisation as the FP64 one's (96 to 382 cells, condition
// numbers 7e2 to 1e9: amplitudes 2e-15 to 2e-11 for both).  All this holds for a positive
// definite matrix; where F is not, its factor outgrows the integers' range, and
// k_chol64_plain takes over.
//
// What bounds it, for one evaluation (tensor pipe 5 %, DRAM nothing): the chain of pivot
// blocks, ~80 us per 64 columns -- 46 us the pivots (0.7 us each: 1/sqrt, two barriers, and wide integer
// multiplies at a quarter of the plain rate), 6 us the inverse's digits, 8 us the
// product below the block, 20 us the way to the next diagonal tile through flags
// and global memory.  2,934 cells: F and R and the solves 43.3 -> 4.2 ms, 738
// cells 7.5 -> 1.1 ms, 96 cells 1.1 -> 0.2 ms (before: 64-wide FP64 kernels, three
// launches per step, R as if it were dense and the solves on one SM).
// Tried, not faster: FP64 in the pivot blocks (76 us a block), the pivots in pairs
// through their 2x2 determinant (registers spill), rows 64-127 of a diagonal
// tile summed while its pivots run (the tile's other steps grew by as much).
#include <cuda_fp16.h>
#include <algorithm>
#include "qlpix_ctx.h"
#include "ozaki.cuh"
#include "tma_map.h"

namespace qlpix {

#define C64 64
#define CS 8                       // digits of the factor
#define CB_STAGE oz_stage_bytes(CS)
#define C64_POISON (1 << 20)       // exponent of a row that holds no finite number: its pivot becomes NaN

struct Chol64Work {
    __half* ls = nullptr;          // [CS][M128][64 wb] digits of the factor, block column k at k mod wb
    __half* li = nullptr;          // [CS][M128][64] digits of the diagonal blocks' inverses
    int* rexp = nullptr;           // [M128] E_i
    int* lexp = nullptr;           // [M128] exponents of the inverses' rows
    int* wexp = nullptr;           // [nbc] the inverses' grids
    int* flags = nullptr;          // ready[nbc][nbc] (column, row block), inverse[nbc], tile counter,
                                   // two solves' [nbc] each, redo (a pivot <= 0), its tile counter
    double* diag = nullptr;        // F's: [M128] its diagonal, for k_chol64_plain
    int M128 = 0, nbc = 0, wb = 0; // wb: block columns kept of a row (all; of a band the band + 2)
    bool own_ls = false;
    CUtensorMap ls_a, ls_b, li_b;
};

__device__ __forceinline__ void bar_sync(int id, int threads)
{
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(threads) : "memory");
}

__device__ __forceinline__ void fence_async() { asm volatile("fence.proxy.async;" ::: "memory"); }

// v 2^e by its exponent bits (v normal or zero, the result normal)
__device__ __forceinline__ double mul_pow2(double v, int e)
{
    return v == 0.0 ? v : __longlong_as_double(__double_as_longlong(v) + ((long long)e << 52));
}

// round(x 2^sh), |result| < 2^62; infinities and NaN give 0 (their rows are marked)
__device__ __forceinline__ long long fx_from_double(double x, int sh)
{
    const long long b = __double_as_longlong(x);
    const int e = (int)((b >> 52) & 0x7ff);
    if (e == 0 || e == 2047) return 0;
    const long long m = (b & 0xfffffffffffffll) | (1ll << 52);
    const int s = e - 1075 + sh;
    long long q;
    if (s >= 0) q = s <= 9 ? (m << s) : (1ll << 62) - 1;
    else q = s > -55 ? ((m + (1ll << (-s - 1))) >> -s) : 0;
    return b < 0 ? -q : q;
}

// k with d 2^-62 = m 4^-k, m in [1/4, 1) (1 for d = 2^62)
__device__ __forceinline__ int fx_scale4(long long d) { return max(0, (__clzll(d) - 2) >> 1); }

// Products of 62-bit numbers by 31-bit halves a = ah 2^31 + al (al >= 0): three
// wide multiplies; al bl is left out, so a product comes out 3/4 of its unit low
// on average.
__device__ __forceinline__ int fx_hi(long long a) { return (int)(a >> 31); }
__device__ __forceinline__ int fx_lo(long long a) { return (int)a & 0x7fffffff; }

// 1/sqrt(d 2^-62) = r 2^-60 2^k, r in (2^60, 2^61], for d in (0, 2^62]: the FP32
// estimate and one step of third order in integers (relative error ~2^-59).
__device__ __forceinline__ void fx_rsqrt(long long d, long long& r, int& k)
{
    k = fx_scale4(d);
    const unsigned long long m = (unsigned long long)d << (2 * k);    // 2^-62
    const float y0 = rsqrtf((float)(int)(m >> 32) * 0x1p-30f);
    const uint32_t y = __float2uint_rz(fminf(y0, 2.0f) * 0x1p30f);   // 2^-30
    const unsigned long long y2 = (unsigned long long)y * y;          // 2^-60
    const uint32_t mh = (uint32_t)(m >> 31), ml = (uint32_t)m & 0x7fffffffu;
    const uint32_t yh = (uint32_t)(y2 >> 31), yl = (uint32_t)y2 & 0x7fffffffu;
    const unsigned long long h = (unsigned long long)mh * yh + (((unsigned long long)mh * yl + (unsigned long long)ml * yh) >> 31);
    const long long e = (1ll << 60) - 1 - (long long)h;               // 1 - m y^2 on 2^-60, |e| < 2^40
    const int es = (int)(e >> 24);                                    // ... on 2^-36
    const long long c = (e >> 1) + ((3ll * ((long long)es * es)) >> 15);   // e / 2 + 3 e^2 / 8
    r = ((long long)y << 30) + (((long long)(int)(c >> 16) * (long long)y) >> 14) + (long long)(((unsigned long long)(c & 0xffff) * y) >> 30);
}

// t r 2^-60 for |t| <= 2^62, r <= 2^61
__device__ __forceinline__ long long fx_mul60(long long t, long long r)
{
    const int th = fx_hi(t), tl = fx_lo(t), rh = fx_hi(r), rl = fx_lo(r);
    return ((long long)th * rh << 2) + (((long long)th * rl + (long long)tl * rh) >> 29);
}

// a b 2^-62
__device__ __forceinline__ long long fx_mul62(long long a, long long b)
{
    const int ah = fx_hi(a), al = fx_lo(a), bh = fx_hi(b), bl = fx_lo(b);
    return (long long)ah * bh + (((long long)ah * bl + (long long)al * bh) >> 31);
}

// x 2^s, saturating at 2^62
__device__ __forceinline__ long long fx_shl(long long x, int s)
{
    const long long top = (1ll << 62) >> s;
    return x > top ? 1ll << 62 : (x < -top ? -(1ll << 62) : x << s);
}

// The diagonal block's factor and inverse (64-bit integers) sit in the A digits'
// rows 0-63 of the two stages, which a diagonal tile's product does not need:
// eight rows of 512 bytes per digit block, the columns rotated against bank
// conflicts of the column-wise stores.
__device__ __forceinline__ long long& diag_at(unsigned char* stage, int i, int c)
{
    return *reinterpret_cast<long long*>(stage + (i >> 3) * OZ_A_BYTES + (i & 7) * 512 + ((c ^ (i & 31)) << 3));
}

struct Diag64 {
    long long col[C64];        // the pivot column before its division, on 2^-62
    int2 y[C64];               // halves of -l_c (2^-62) right of the pivot, of minus the inverse's row (2^-58) up to it
    int2 l[C64];               // halves of the pivot column of the factor, on 2^-62
    long long brow[C64];       // the pivot's row of the inverse before its division, on 2^-58
    int g[C64];                // the block's own scaling: row and column i times 2^g_i
    int first_bad;             // first negative pivot + 1, 0 none
    int redo;                  // a pivot that is not positive
    int wide;                  // the inverse left its range: redone in FP64
    int w;                     // it is kept on 2^-(58 - w)
    int top;                   // bits of its largest entry
};
#define D64_TOP ((1ll << 62) - 1)   // bound on the factor's entries (1 on 2^-62) and the inverse's (16 on 2^-58)

__device__ __forceinline__ int2 fx_halves(long long x) { return make_int2(fx_hi(x), fx_lo(x)); }

// Steps 16 P .. 16 P + 15 of the 64x64 block held by 256 threads: thread (ty, tx)
// = (tid / 16, tid % 16) owns the entries (ty + 16 u, tx + 16 v), u >= v.  An
// entry right of the pivot column is the Schur complement (2^-62); once its
// column has been the pivot it is the inverse's row before its final division
// (2^-58): the column of L times the pivot's finished row of the inverse is
// subtracted from it, the forward substitution on the identity, run along with
// the factorisation.  Either way an entry loses l_i y_c.  A step is two
// barriers: the column and the inverse's row divided (64 threads each, all forming
// 1/sqrt of the pivot), then every entry updated.  What the products lose on
// average (3/4 of a unit a step) is put back where an entry is used.
template <int P>
__device__ __forceinline__ void diag64_steps(long long (&q)[10], Diag64& s, unsigned char* L, unsigned char* X,
                                             const int* poison)
{
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    int big = 0;                              // sign bit: an entry passed 2^62 (it grows by less than 2^62 a step)
    #pragma unroll 1
    for (int jj = 0; jj < 16; jj++) {
        const int j = 16 * P + jj;
        if (tid < 128) {
            const int i = tid & 63;
            long long d = s.col[j] + ((3 * j) >> 2), r;
            const long long t = tid < 64 ? (i == j ? (d < 0 ? -d : d) : s.col[i] + ((3 * j) >> 2))
                                         : s.brow[i] + ((3 * (j - i)) >> 2);
            int k;
            if (tid == 0 && (d <= 0 || poison[j])) s.redo = 1;
            if (d < 0) {
                if (tid == 0 && s.first_bad == 0 && !poison[j]) s.first_bad = j + 1;
                d = -d;
            }
            fx_rsqrt(min(max(d, 1ll), D64_TOP), r, k);
            if (tid < 64) {
                if (i >= j) {
                    const long long l = min(max(fx_mul60(t << k, r), -D64_TOP), D64_TOP);
                    s.l[i] = fx_halves(l);
                    if (i > j) s.y[i] = fx_halves(-l);
                    diag_at(L, i, j) = l;
                }
            } else {
                long long x = 0;
                if (i < j) {
                    if ((t < 0 ? -t : t) > D64_TOP >> k) s.wide = 1;
                    x = fx_mul60(t << k, r);
                } else if (i == j) {
                    if (k >= 3 + s.w) s.wide = 1;
                    x = (r >> (2 + s.w)) << k;
                }
                if (x > D64_TOP || x < -D64_TOP) s.wide = 1;
                if (i <= j) s.y[i] = fx_halves(-x);
                diag_at(X, j, i) = x;
            }
        }
        bar_sync(1, 256);
        int2 y[4];
        #pragma unroll
        for (int v = 0; v < 4; v++) y[v] = s.y[tx + 16 * v];
        #pragma unroll
        for (int u = P; u < 4; u++) {
            const int i = ty + 16 * u;
            if (i <= j) continue;
            const int2 l = s.l[i];
            #pragma unroll
            for (int v = 0; v <= u; v++) {
                const int c = tx + 16 * v;
                long long& e = q[u * (u + 1) / 2 + v];
                if (v == P && c == j) e = 0;
                const long long lo = (long long)l.x * y[v].y + (long long)l.y * y[v].x;
                e += (long long)l.x * y[v].x;
                e += lo >> 31;
                const int top = (int)(e >> 32);
                big |= top ^ (top << 1);
                if (v >= P && c == j + 1) s.col[i] = e;
                if (v <= P && c <= j && i == j + 1) s.brow[c] = e;
            }
        }
        if (jj == 15 && big < 0) s.wide = 1;
        bar_sync(1, 256);
    }
}

// A block whose inverse leaves the integers' range (the first of an
// ill-conditioned matrix; the next ones take their grid from it): formed in FP64 from the factor, one row of the inverse a step and
// its outer product with the factor's column taken off the rows below, then
// back to integers on a grid that holds the largest entry.
__device__ __noinline__ void diag64_wide(Diag64& s, unsigned char* L, unsigned char* X)
{
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    double* row = reinterpret_cast<double*>(s.y);
    double* col = reinterpret_cast<double*>(s.l);
    double e[16], big = 0;
    #pragma unroll
    for (int k = 0; k < 16; k++) e[k] = 0;                   // (ty + 16 u, tx + 16 v) at 4 u + v
    #pragma unroll 1
    for (int j = 0; j < C64; j++) {
        #pragma unroll
        for (int u = 0; u < 4; u++)
            if (ty + 16 * u == j) {
                const double r = 1.0 / fmax((double)diag_at(L, j, j) * 0x1p-62, 0x1p-62);
                #pragma unroll
                for (int v = 0; v < 4; v++) {
                    const int c = tx + 16 * v;
                    const double x = c < j ? e[4 * u + v] * r : (c == j ? r : 0.0);
                    row[c] = x;
                    diag_at(X, j, c) = __double_as_longlong(x);
                    big = fmax(big, fabs(x));
                }
            }
        if (tid < C64 && tid > j) col[tid] = (double)diag_at(L, tid, j) * 0x1p-62;
        bar_sync(1, 256);
        #pragma unroll
        for (int u = 0; u < 4; u++)
            if (ty + 16 * u > j)
                #pragma unroll
                for (int v = 0; v <= u; v++) e[4 * u + v] -= col[ty + 16 * u] * row[tx + 16 * v];
        bar_sync(1, 256);
    }
    if (tid == 0) s.w = 0;
    bar_sync(1, 256);
    atomicMax(&s.w, max(0, (int)((__double_as_longlong(big) >> 52) & 0x7ff) - 1023 + 1 - 4));
    bar_sync(1, 256);
    const double scale = exp2((double)(58 - s.w));
    #pragma unroll
    for (int k = 0; k < 16; k++) {
        long long& x = diag_at(X, ty + 16 * (k >> 2), tx + 16 * (k & 3));
        x = __double2ll_rn(__longlong_as_double(x) * scale);
    }
    bar_sync(1, 256);
}

// E_i from the diagonal: sqrt(F_ii) < 2^E_i.
__global__ void k_chol64_prep(const GridState* __restrict__ gs, const double* __restrict__ F, int ld,
                              int* __restrict__ rexp)
{
    const int Mp = (gs->M + 63) & ~63;
    for (int i = blockIdx.x * blockDim.x + threadIdx.x; i < Mp; i += gridDim.x * blockDim.x) {
        const int e = oz_exponent(F[(size_t)i * ld + i]);
        rexp[i] = (e == 0 || e == 2047) ? C64_POISON : (e - 1021) >> 1;
    }
}

// Waits (bounded) until *p is set; gives up early when another CTA did.
__device__ __forceinline__ bool wait_flag(const int* p, GridState* gs, volatile int* abort_flag)
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

// band: blocks below the diagonal that can be nonzero, even (a tile's second
// 64 rows reach one further); dense: any number past the matrix.  Nothing reads a row's
// block column k once its column k + band + 2 stands, so a band's digits turn round in
// wb = band + 2 block columns (all of them were 0.27 GB a slot at 4,096 cells, now 17 MB).
// linv: the inverses of the diagonal blocks in FP64 for the solves, or null.
// redo, diag0 (F; R is positive definite by construction: null): the matrix is kept
// above its diagonal and in diag0, and *redo set where a pivot is not positive, for
// k_chol64_plain.
__global__ void __launch_bounds__(OZ_THREADS, 1) k_chol64(const __grid_constant__ CUtensorMap ls_a,
                                                         const __grid_constant__ CUtensorMap ls_b,
                                                         const __grid_constant__ CUtensorMap li_b, GridState* gs,
                                                         double* F, int ld, int which, int band, int M128, int nbc, int wb,
                                                         __half* ls, __half* li, const int* rexp, int* lexp,
                                                         int* wexp, int* flags, double* linv, int* redo,
                                                         double* diag0)
{
    extern __shared__ unsigned char smem_raw[];
    __shared__ OzPipe pipe;
    __shared__ Diag64 dg;
    __shared__ uint64_t b_full;
    __shared__ int ticket;
    __shared__ int row_e[OZ_TM], col_e[C64], bits[2][OZ_TM], poison[C64];
    const int Mp = (gs->M + 63) & ~63, nb = Mp / C64;
    int* ready = flags;
    int* inv = flags + (size_t)nbc * nbc;
    int* counter = inv + nbc;
    unsigned char* smem = (unsigned char*)(((uintptr_t)smem_raw + 1023) & ~(uintptr_t)1023);
    unsigned char* const SL = smem;                    // the diagonal block's factor (diag_at)
    unsigned char* const SX = smem + CB_STAGE;         // ... and its inverse
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) mbar_init(&b_full, 1);
    oz_begin(pipe);

    int it0 = 0, f0 = 0, nb_full = 0;            // stages, accumulator readings, loads on b_full so far
    int j = 0, base = 0;                         // the current ticket's column; the tickets before that column
    while (true) {
        if (threadIdx.x == 0) ticket = atomicAdd(counter, 1);
        __syncthreads();
        const int tk = ticket;
        auto tiles_of = [&](int c) { return min((nb - c + 1) >> 1, (band >> 1) + 1); };
        while (j < nb && tk >= base + tiles_of(j)) { base += tiles_of(j); j++; }
        if (j >= nb) break;
        const int t = tk - base, rb = j + 2 * t;
        const int k0 = max(0, rb - band), n = 2 * (j - k0);
        const bool second = rb + 1 < nb;         // the tile's rows 64..127 exist
        const bool solve = t > 0 || second;
        if (threadIdx.x < OZ_TM) {
            const int row = rb * C64 + threadIdx.x;
            row_e[threadIdx.x] = row < Mp ? (rexp[row] == C64_POISON ? 0 : rexp[row]) : 0;
        } else if (threadIdx.x < OZ_TM + C64) {
            const int e = rexp[j * C64 + threadIdx.x - OZ_TM];
            col_e[threadIdx.x - OZ_TM] = e == C64_POISON ? 0 : e;
            poison[threadIdx.x - OZ_TM] = e == C64_POISON;
        }
        if (threadIdx.x == 0) dg.first_bad = dg.redo = dg.wide = dg.top = dg.w = 0;
        __syncthreads();

        const int r = 32 * (warp & 3) + lane, h = (warp >> 2) & 1;       // an epilogue thread's row and column half
        const int row = rb * C64 + r;
        long long hi[32];
        uint32_t lo[32];
        // ---- the Schur complement: F_ij - sum_k L_ik L_jk^T ----
        if (warp == OZ_EPI) {
            if (lane == 0) {
                for (int k = k0; k < j; k++) {
                    const int* rk = ready + (size_t)k * nbc;
                    if (!wait_flag(rk + rb, gs, &pipe.abort) || !wait_flag(rk + j, gs, &pipe.abort) ||
                        (second && !wait_flag(rk + rb + 1, gs, &pipe.abort)))
                        break;
                    fence_async();
                    bool ok = true;
                    for (int half = 0; half < 2 && ok; half++) {
                        const int it = it0 + 2 * (k - k0) + half;
                        ok = oz_load_stage<CS>(pipe, smem, it, &ls_a, &ls_b, M128, (k % wb) * C64 + half * OZ_KS, rb * C64,
                                               j * C64);
                        if (ok) pipe.n_issued = it + 1;
                    }
                    if (!ok) break;
                }
            }
            __syncwarp();
        } else if (warp == OZ_EPI + 1) {
            if (lane == 0) oz_mma_loop<CS>(pipe, smem, it0, f0, n);
            __syncwarp();
        } else {
            const double* src = F + (size_t)row * ld + j * C64 + 32 * h;
            double* up = F + (size_t)(j * C64 + 32 * h) * ld + row;       // (the diagonal block's: below)
            const bool keep = redo && row < Mp && (t > 0 || r >= C64);
            #pragma unroll
            for (int c = 0; c < 32; c += 2) {
                double2 a = make_double2(0.0, 0.0);
                if (row < Mp) a = *reinterpret_cast<const double2*>(src + c);
                if (keep) { up[(size_t)c * ld] = a.x; up[(size_t)(c + 1) * ld] = a.y; }
                const long long v0 = -fx_from_double(a.x, 60 - row_e[r] - col_e[32 * h + c]);
                const long long v1 = -fx_from_double(a.y, 60 - row_e[r] - col_e[32 * h + c + 1]);
                hi[c] = v0 >> 24; lo[c] = (uint32_t)v0 << 8;             // v 2^8 = hi 2^32 + lo on 2^-68
                hi[c + 1] = v1 >> 24; lo[c + 1] = (uint32_t)v1 << 8;
            }
            oz_accumulate<CS>(pipe, f0, n, hi, lo);
            #pragma unroll
            for (int c = 0; c < 32; c++)
                hi[c] = -((hi[c] << 24) + (long long)((lo[c] >> 8) + ((lo[c] >> 7) & 1)));      // rounded to 2^-60
        }
        it0 += n;
        f0 += (n + OZ_FLUSH - 1) / OZ_FLUSH;
        __syncthreads();                          // every MMA has read its stage: the buffers are free

        if (warp < OZ_EPI) {
            const int tid = threadIdx.x;
            if (t == 0) {
                // ---- the diagonal block: factor and inverse ----
                // scaled so that its diagonal lies in [1/4, 1): its inverse then
                // is that of a matrix near a correlation matrix
                if (r < C64 && (r >> 5) == h) {
                    long long d = 1;
                    #pragma unroll
                    for (int c = 0; c < 32; c++) d = (c == (r & 31)) ? hi[c] : d;
                    dg.g[r] = fx_scale4(max(d << 2, 1ll));
                }
                // the inverse's grid from the size of the last one, which the sums
                // waited for
                if (tid == 0 && j > 0) dg.w = __ldcg(wexp + j - 1);
                bar_sync(1, 256);
                if (r < C64) {
                    #pragma unroll
                    for (int c = 0; c < 32; c++) {
                        const long long v = fx_shl(hi[c], 2 + dg.g[r] + dg.g[32 * h + c]);
                        diag_at(SL, r, 32 * h + c) = v;
                        if (c == 0 && h == 0) dg.col[r] = v;
                    }
                }
                bar_sync(1, 256);
                {
                    long long q[10];
                    const int tx = tid & 15, ty = tid >> 4;
                    #pragma unroll
                    for (int u = 0; u < 4; u++)
                        #pragma unroll
                        for (int v = 0; v <= u; v++)
                            q[u * (u + 1) / 2 + v] = diag_at(SL, ty + 16 * u, tx + 16 * v);
                    bar_sync(1, 256);
                    diag64_steps<0>(q, dg, SL, SX, poison);
                    diag64_steps<1>(q, dg, SL, SX, poison);
                    diag64_steps<2>(q, dg, SL, SX, poison);
                    diag64_steps<3>(q, dg, SL, SX, poison);
                }
                if (dg.wide) diag64_wide(dg, SL, SX);
                // the inverse's digits for the rows below: 4 threads a row; entry
                // (c, m) undoes the block's scaling of column m (2^g_m)
                {
                    const int c = tid >> 2, m0 = (tid & 3) * 16;
                    long long x[16];
                    int e = -4096, big = 0;       // bits of the row's largest entry, and without the scaling
                    #pragma unroll
                    for (int m = 0; m < 16; m++) {
                        x[m] = diag_at(SX, c, m0 + m);
                        const int bits = 64 - __clzll(x[m] < 0 ? -x[m] : x[m]);
                        big = max(big, bits);
                        if (x[m]) e = max(e, bits + dg.g[m0 + m]);
                    }
                    e = max(e, __shfl_xor_sync(0xffffffffu, e, 1));
                    e = max(e, __shfl_xor_sync(0xffffffffu, e, 2));
                    for (int o = 1; o < 32; o <<= 1) big = max(big, __shfl_xor_sync(0xffffffffu, big, o));
                    if (lane == 0) atomicMax(&dg.top, big);
                    const int sh = oz_bits(CS) - e;
                    unsigned long long b[16];
                    #pragma unroll
                    for (int m = 0; m < 16; m++) {
                        const int sm = sh + dg.g[m0 + m];
                        b[m] = oz_bias<CS>(sm >= 0 ? x[m] << min(sm, 62) : (x[m] + (1ll << (min(-sm, 63) - 1))) >> min(-sm, 63));
                    }
                    #pragma unroll
                    for (int d = 0; d < CS; d++)
                        #pragma unroll
                        for (int w = 0; w < 2; w++)
                            *reinterpret_cast<uint4*>(li + ((size_t)d * M128 + j * C64 + c) * C64 + m0 + 8 * w) =
                                oz_digits8<CS>(b + 8 * w, d);
                    // x 2^-(58 - w) = (x 2^sh) 2^(E - 62)
                    if ((tid & 3) == 0) lexp[j * C64 + c] = 4 + dg.w - sh;
                    fence_async();
                    bar_sync(1, 256);
                    if (tid == 0) {
                        wexp[j] = min(40, max(0, dg.w + dg.top - 60));       // two bits to spare in the next one
                        st_release(inv + j, 1);
                    }
                    unsigned char* bs = smem + (m0 >> 5) * CB_STAGE + CS * OZ_A_BYTES;
                    #pragma unroll
                    for (int d = 0; d < CS; d++)
                        #pragma unroll
                        for (int w = 0; w < 2; w++)
                            *reinterpret_cast<uint4*>(bs + d * OZ_B_BYTES + oz_chunk(c, ((m0 & 31) >> 3) + w)) =
                                oz_digits8<CS>(b + 8 * w, d);
                }
            }
            if (solve) {
                // ---- the rows below the diagonal block: times the inverse, transposed ----
                long long mx = 0;
                #pragma unroll
                for (int c = 0; c < 32; c++) mx |= hi[c] < 0 ? -hi[c] : hi[c];
                bits[h][r] = 64 - __clzll(mx);
                bar_sync(1, 256);
                const int nbit = max(bits[0][r], bits[1][r]);
                const int sh = nbit ? max(0, oz_bits(CS) - nbit) : 0;      // T 2^sh, at most 2^62
                const bool mine = row < Mp && (t > 0 || r >= C64);
                if (mine) {
                    unsigned char* as = smem + h * CB_STAGE;
                    unsigned long long b[8];
                    #pragma unroll
                    for (int w = 0; w < 4; w++) {
                        #pragma unroll
                        for (int c = 0; c < 8; c++) b[c] = oz_bias<CS>(hi[8 * w + c] << sh);
                        #pragma unroll
                        for (int d = 0; d < CS; d++)
                            *reinterpret_cast<uint4*>(as + d * OZ_A_BYTES + oz_chunk(r, w)) = oz_digits8<CS>(b, d);
                    }
                }
                fence_async();
                bar_sync(2, 32 * (OZ_EPI + 1));
                #pragma unroll
                for (int c = 0; c < 32; c++) { hi[c] = 0; lo[c] = 0; }
                oz_accumulate<CS>(pipe, f0, 2, hi, lo);
                if (mine) {
                    // (hi 2^32 + lo) 2^(2 - sh + e_col - 68), kept on 2^-62
                    #pragma unroll
                    for (int c = 0; c < 32; c++) {
                        const int s = sh + 4 - __ldcg(lexp + j * C64 + 32 * h + c);        // to the right
                        const __int128 V = ((__int128)hi[c] << 32) + lo[c];
                        const long long x = s > 0 ? (long long)(V >> (s - 1)) : (long long)(V << (min(-s, 60) + 1));
                        hi[c] = min(max((x + 1) >> 1, -(1ll << oz_bits(CS))), 1ll << oz_bits(CS));
                    }
                    __half* out = ls + (size_t)row * wb * C64 + (j % wb) * C64 + 32 * h;
                    unsigned long long b[8];
                    #pragma unroll
                    for (int w = 0; w < 4; w++) {
                        #pragma unroll
                        for (int c = 0; c < 8; c++) b[c] = oz_bias<CS>(hi[8 * w + c]);
                        #pragma unroll
                        for (int d = 0; d < CS; d++)
                            *reinterpret_cast<uint4*>(out + (size_t)d * M128 * wb * C64 + 8 * w) = oz_digits8<CS>(b, d);
                    }
                }
                fence_async();
                bar_sync(1, 256);
                if (tid == 0 && !pipe.abort) {
                    int* rj = ready + (size_t)j * nbc + rb;
                    if (t > 0) st_release(rj, 1);
                    if (second) st_release(rj + 1, 1);
                }
                if (mine) {
                    double* dst = F + (size_t)row * ld + j * C64 + 32 * h;
                    const int e = row_e[r] - oz_bits(CS);
                    #pragma unroll
                    for (int c = 0; c < 32; c += 2)
                        *reinterpret_cast<double2*>(dst + c) = make_double2(mul_pow2((double)hi[c], e),
                                                                            mul_pow2((double)hi[c + 1], e));
                }
            }
            if (t == 0) {
                // the factor's diagonal block and its inverse in FP64: nothing in
                // this launch reads them
                if (redo) {
                    double a[16];
                    #pragma unroll
                    for (int u = 0; u < 16; u++) a[u] = F[(size_t)(j * C64 + u * 4 + (tid >> 6)) * ld + j * C64 + (tid & 63)];
                    #pragma unroll
                    for (int u = 0; u < 16; u++) {
                        const int i = u * 4 + (tid >> 6), c = tid & 63;
                        if (c < i) F[(size_t)(j * C64 + c) * ld + j * C64 + i] = a[u];
                        if (c == i) diag0[j * C64 + i] = a[u];
                    }
                    if (tid == 0 && dg.redo) *redo = 1;
                }
                for (int u = 0; u < 16; u++) {
                    const int i = u * 4 + (tid >> 6), c = tid & 63;
                    if (c <= i) {
                        double v = mul_pow2((double)diag_at(SL, i, c), col_e[i] - dg.g[i] - 62);
                        if (i == c && (poison[i] || v == 0.0)) v = __longlong_as_double(0x7ff8000000000000ll);
                        F[(size_t)(j * C64 + i) * ld + j * C64 + c] = v;
                    }
                    if (linv)
                        linv[(size_t)(j * C64 + i) * C64 + c] =
                            c <= i ? mul_pow2((double)diag_at(SX, i, c), dg.w - 58 + dg.g[c] - col_e[c]) : 0.0;
                }
                if (tid == 0 && dg.first_bad && !redo) {
                    int* flag = which ? &gs->not_spd_R : &gs->not_spd_F;
                    if (*flag == 0) *flag = j * C64 + dg.first_bad;
                }
            }
        } else if (warp == OZ_EPI) {
            if (t > 0) {
                if (lane == 0 && wait_flag(inv + j, gs, &pipe.abort)) {
                    fence_async();
                    mbar_expect_tx(&b_full, 2 * CS * OZ_B_BYTES);
                    for (int half = 0; half < 2; half++)
                        for (int d = 0; d < CS; d++)
                            tma_load_2d(&li_b, &b_full, smem + half * CB_STAGE + CS * OZ_A_BYTES + d * OZ_B_BYTES,
                                        half * OZ_KS, d * M128 + j * C64);
                    // landed before the buffers are used again, whatever the others do
                    mbar_wait_bounded(&b_full, nb_full & 1, &pipe.abort, false);
                }
            }
            __syncwarp();
        } else {
            if (solve) {
                bar_sync(2, 32 * (OZ_EPI + 1));
                if (lane == 0 && (t == 0 || mbar_wait_bounded(&b_full, nb_full & 1, &pipe.abort))) {
                    tc_fence_after();
                    oz_mma_filled<CS>(pipe, smem, f0);
                }
                __syncwarp();
            }
        }
        if (solve) f0++;
        if (t > 0) nb_full++;
        // the one place to leave early: behind a barrier nobody raises pipe.abort until the next one (a
        // thread that saw it raised by a faster warp's wait would leave the others at their barriers)
        __syncthreads();
        if (pipe.abort) break;
    }
    if (threadIdx.x == 32 * (OZ_EPI + 1)) mma_commit(&pipe.done);
    __syncwarp();
    oz_end(pipe);
    if (pipe.abort && threadIdx.x == 0) atomicExch(&gs->status, QLP_ERR_TIMEOUT);
}

// ---------------------------------------------------------------------------
// F = L L^T in FP64, where k_chol64 met a pivot that is not positive (or a row that
// holds no finite number): sqrt(|d|) at a negative one, flagged, and no bound on what
// follows, as the reference goes on.  Left-looking over 64x64 tiles from a counter, as
// k_chol64, the same flags with the value 2; the matrix comes from above the
// diagonal and diag0.  Bound by the FP64 pipe (M^3 / 3 multiply-adds at 2 a clock and
// SM); nothing but the look at *redo for any other matrix.
// ---------------------------------------------------------------------------
#define CP_SMEM (2 * C64 * (C64 + 1) * (int)sizeof(double))

// All threads wait (bounded) until *p and *q are 2.
__device__ __forceinline__ bool wait_redone(const int* p, const int* q, GridState* gs, int* sh)
{
    if (threadIdx.x == 0) {
        const uint64_t t0 = globaltimer();
        bool ok;
        while (!(ok = ld_acquire(p) == 2 && ld_acquire(q) == 2)) {
            if (*(volatile int*)&gs->status == QLP_ERR_TIMEOUT || globaltimer() - t0 > TC_WAIT_NS) break;
            __nanosleep(64);
        }
        if (!ok) atomicExch(&gs->status, QLP_ERR_TIMEOUT);
        *sh = ok ? 1 : 0;
    }
    __syncthreads();
    const bool ok = *sh != 0;
    __syncthreads();
    return ok;
}

__global__ void __launch_bounds__(256) k_chol64_plain(GridState* gs, double* F, int ld, const double* diag0, int nbc,
                                                      int* flags, const int* redo, int* counter, double* linv)
{
    if (*redo == 0) return;
    extern __shared__ double cp_smem[];
    __shared__ double colj[C64];
    __shared__ int sh, ticket;
    double (*P)[C64 + 1] = reinterpret_cast<double (*)[C64 + 1]>(cp_smem);
    double (*Q)[C64 + 1] = reinterpret_cast<double (*)[C64 + 1]>(cp_smem + C64 * (C64 + 1));
    const int nb = ((gs->M + 63) & ~63) / C64;
    int* ready = flags;
    int* inv = flags + (size_t)nbc * nbc;
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    int j = 0, base = 0;
    while (true) {
        if (tid == 0) ticket = atomicAdd(counter, 1);
        __syncthreads();
        const int tk = ticket;
        __syncthreads();
        while (j < nb && tk >= base + nb - j) { base += nb - j; j++; }
        if (j >= nb) return;
        const int i = j + tk - base;
        const bool diag = i == j;
        double acc[4][4];
        #pragma unroll
        for (int u = 0; u < 4; u++)
            #pragma unroll
            for (int v = 0; v < 4; v++) {
                const int r = ty * 4 + u, c = tx * 4 + v;
                acc[u][v] = (diag && r == c) ? diag0[j * C64 + r]
                            : (diag && r < c) ? 0.0 : F[(size_t)(j * C64 + c) * ld + i * C64 + r];
            }
        for (int k = 0; k < j; k++) {
            const int* rk = ready + (size_t)k * nbc;
            if (!wait_redone(rk + i, rk + j, gs, &sh)) return;
            for (int e = tid; e < C64 * C64; e += 256) {
                const int r = e >> 6, m = e & 63;
                P[r][m] = __ldcg(F + (size_t)(i * C64 + r) * ld + k * C64 + m);
                Q[r][m] = __ldcg(F + (size_t)(j * C64 + r) * ld + k * C64 + m);
            }
            __syncthreads();
            #pragma unroll 4
            for (int m = 0; m < C64; m++) {
                double a[4], b[4];
                #pragma unroll
                for (int u = 0; u < 4; u++) { a[u] = P[ty * 4 + u][m]; b[u] = Q[tx * 4 + u][m]; }
                #pragma unroll
                for (int u = 0; u < 4; u++)
                    #pragma unroll
                    for (int v = 0; v < 4; v++) acc[u][v] -= a[u] * b[v];
            }
            __syncthreads();
        }
        #pragma unroll
        for (int u = 0; u < 4; u++)
            #pragma unroll
            for (int v = 0; v < 4; v++) P[ty * 4 + u][tx * 4 + v] = acc[u][v];
        if (diag) {
            __syncthreads();
            for (int p = 0; p < C64; p++) {
                if (tid >= p && tid < C64) {
                    const double d = P[p][p], sd = sqrt(fabs(d));
                    if (tid == p && d < 0) atomicCAS(&gs->not_spd_F, 0, j * C64 + p + 1);
                    colj[tid] = tid == p ? sd : P[tid][p] / sd;
                }
                __syncthreads();
                for (int r = p + 1 + ty; r < C64; r += 16) {
                    const double l = colj[r];
                    for (int c = p + 1 + tx; c <= r; c += 16) P[r][c] -= l * colj[c];
                }
                if (tid >= p && tid < C64) P[tid][p] = colj[tid];
                __syncthreads();
            }
            // the inverse, four threads a column
            const int c = tid >> 2, q = tid & 3;
            for (int r = 0; r < C64; r++) {
                double part = 0;
                if (r > c)
                    for (int m = c + q; m < r; m += 4) part += P[r][m] * Q[m][c];
                part += __shfl_xor_sync(0xffffffffu, part, 1);
                part += __shfl_xor_sync(0xffffffffu, part, 2);
                if (q == 0) Q[r][c] = r < c ? 0.0 : (r == c ? 1.0 / P[r][r] : -part / P[r][r]);
                __syncwarp();
            }
            __syncthreads();
            for (int e = tid; e < C64 * C64; e += 256) {
                const int r = e >> 6, m = e & 63;
                if (m <= r) F[(size_t)(j * C64 + r) * ld + j * C64 + m] = P[r][m];
                linv[(size_t)(j * C64 + r) * C64 + m] = Q[r][m];
            }
        } else {
            if (!wait_redone(inv + j, inv + j, gs, &sh)) return;
            // by substitution (a product with the block's inverse loses digits where the
            // factor grows), four threads a row
            for (int e = tid; e < C64 * C64; e += 256) {
                const int r = e >> 6, m = e & 63;
                if (m <= r) Q[r][m] = __ldcg(F + (size_t)(j * C64 + r) * ld + j * C64 + m);
            }
            __syncthreads();
            const int r = tid >> 2, q = tid & 3;
            for (int c = 0; c < C64; c++) {
                double part = 0;
                for (int m = q; m < c; m += 4) part += P[r][m] * Q[c][m];
                part += __shfl_xor_sync(0xffffffffu, part, 1);
                part += __shfl_xor_sync(0xffffffffu, part, 2);
                if (q == 0) P[r][c] = (P[r][c] - part) / Q[c][c];
                __syncwarp();
            }
            __syncthreads();
            for (int e = tid; e < C64 * C64; e += 256)
                F[(size_t)(i * C64 + (e >> 6)) * ld + j * C64 + (e & 63)] = P[e >> 6][e & 63];
        }
        __threadfence();
        __syncthreads();
        if (tid == 0) st_release(diag ? inv + j : ready + (size_t)j * nbc + i, 2);
    }
}

// ---------------------------------------------------------------------------
// F z = r with the factor and the inverses of its 64x64 diagonal blocks:
//   forward  y_k = Linv_k (r_k - sum_{j<k} L_kj y_j)
//   backward z_k = Linv_k^T (y_k - sum_{j>k} L_jk^T z_j)
// One CTA per block (the scheme of k_trsv128_fwd / _bwd): CTA k folds in block
// j as soon as its flag is up, so all but the last term of each sum are off the
// critical path, and the FP64 work spreads over the SMs (one CTA ran both sweeps
// before: 4 M^2 FLOP on one SM's FP64 pipe, 2 ms for 2,934 cells).  A thread
// takes 16 terms of a row; its part of the next block and of the inverse is
// loaded before the wait.
// ---------------------------------------------------------------------------
__device__ __forceinline__ bool wait_block(const int* p, GridState* gs, int* sh)
{
    if (threadIdx.x == 0) {
        volatile int stop = 0;
        *sh = wait_flag(p, gs, &stop) ? 1 : 0;
        if (*sh == 0) atomicExch(&gs->status, QLP_ERR_TIMEOUT);
    }
    __syncthreads();
    const bool ok = *sh != 0;
    __syncthreads();
    return ok;
}

__global__ void __launch_bounds__(256) k_trsv64_fwd(const double* __restrict__ L, int ld,
                                                    const double* __restrict__ Linv, GridState* gs,
                                                    const double* __restrict__ r, double* y, int* flags)
{
    __shared__ double t[C64], red[4][C64];
    __shared__ int sh;
    const int nb = ((gs->M + 63) & ~63) / C64, k = blockIdx.x;
    if (k >= nb) return;
    const int row = threadIdx.x & 63, c0 = (threadIdx.x >> 6) * 16;
    const double2* Lr = reinterpret_cast<const double2*>(Linv + (size_t)(k * C64 + row) * C64 + c0);
    double2 lv[8];
    #pragma unroll
    for (int u = 0; u < 8; u++) lv[u] = Lr[u];
    double acc = 0;
    for (int j = 0; j < k; j++) {
        const double2* p = reinterpret_cast<const double2*>(L + (size_t)(k * C64 + row) * ld + j * C64 + c0);
        double2 lp[8];
        #pragma unroll
        for (int u = 0; u < 8; u++) lp[u] = p[u];
        if (!wait_block(flags + j, gs, &sh)) return;
        const double2* yp = reinterpret_cast<const double2*>(y + j * C64 + c0);
        #pragma unroll
        for (int u = 0; u < 8; u++) {
            const double2 v = __ldcg(yp + u);
            acc += lp[u].x * v.x;
            acc += lp[u].y * v.y;
        }
    }
    red[c0 >> 4][row] = acc;
    __syncthreads();
    if (threadIdx.x < C64) {
        const int i = k * C64 + row;
        t[row] = (i < gs->M ? r[i] : 0.0) - ((red[0][row] + red[1][row]) + (red[2][row] + red[3][row]));
    }
    __syncthreads();
    acc = 0;
    #pragma unroll
    for (int u = 0; u < 8; u++) { acc += lv[u].x * t[c0 + 2 * u]; acc += lv[u].y * t[c0 + 2 * u + 1]; }
    red[c0 >> 4][row] = acc;
    __syncthreads();
    if (threadIdx.x < C64) y[k * C64 + row] = (red[0][row] + red[1][row]) + (red[2][row] + red[3][row]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) st_release(flags + k, 1);
}

__global__ void __launch_bounds__(256) k_trsv64_bwd(const double* __restrict__ L, int ld,
                                                    const double* __restrict__ Linv, GridState* gs,
                                                    const double* __restrict__ y, double* z, int* flags)
{
    __shared__ double t[C64], red[4][C64];
    __shared__ int sh;
    const int nb = ((gs->M + 63) & ~63) / C64;
    if ((int)blockIdx.x >= nb) return;
    const int k = nb - 1 - blockIdx.x;
    const int col = threadIdx.x & 63, m0 = (threadIdx.x >> 6) * 16;
    double lv[16];
    #pragma unroll
    for (int u = 0; u < 16; u++) lv[u] = Linv[(size_t)(k * C64 + m0 + u) * C64 + col];
    double acc = 0;
    for (int j = nb - 1; j > k; j--) {
        double lp[16];
        #pragma unroll
        for (int u = 0; u < 16; u++) lp[u] = L[(size_t)(j * C64 + m0 + u) * ld + k * C64 + col];
        if (!wait_block(flags + j, gs, &sh)) return;
        #pragma unroll
        for (int u = 0; u < 16; u++) acc += lp[u] * __ldcg(z + j * C64 + m0 + u);
    }
    red[m0 >> 4][col] = acc;
    __syncthreads();
    if (threadIdx.x < C64)
        t[col] = y[k * C64 + col] - ((red[0][col] + red[1][col]) + (red[2][col] + red[3][col]));
    __syncthreads();
    acc = 0;
    #pragma unroll
    for (int u = 0; u < 16; u++) acc += lv[u] * t[m0 + u];
    red[m0 >> 4][col] = acc;
    __syncthreads();
    if (threadIdx.x < C64) z[k * C64 + col] = (red[0][col] + red[1][col]) + (red[2][col] + red[3][col]);
    __threadfence();
    __syncthreads();
    if (threadIdx.x == 0) st_release(flags + k, 1);
}

// ---------------------------------------------------------------------------
void chol64_free(Chol64Work* z)
{
    if (!z) return;
    void* ptrs[] = {z->own_ls ? z->ls : nullptr, z->li, z->rexp, z->lexp, z->wexp, z->flags, z->diag};
    for (void* p : ptrs) if (p) cudaFree(p);
    delete z;
}

static size_t chol64_flags(const Chol64Work* z) { return (size_t)z->nbc * z->nbc + 3 * z->nbc + 3; }

// Blocks that a band of half_width entries can reach, rounded up to even.
static int chol64_band(int half_width, int M) { return ((std::min(half_width, M) + C64 - 1) / C64 + 1) & ~1; }

// shared: M128 x M128 digits that nothing else uses while this matrix is
// factored (F: the digits of L', read by then), or null to allocate them (R: for
// bands of up to half_width entries).
int chol64_alloc(Chol64Work** out, int M_cap, void* shared, int half_width)
{
    Chol64Work* z = new Chol64Work();
    z->M128 = (M_cap + OZ_TM - 1) / OZ_TM * OZ_TM;
    z->nbc = z->M128 / C64;
    z->own_ls = shared == nullptr;
    z->wb = z->own_ls ? std::min(z->nbc, chol64_band(half_width, M_cap) + 2) : z->nbc;
    z->ls = reinterpret_cast<__half*>(shared);
    cudaError_t e = cudaSuccess;
    auto A = [&](void** p, size_t bytes) { if (e == cudaSuccess) e = cudaMalloc(p, bytes); };
    const size_t rows = (size_t)CS * z->M128;
    if (z->own_ls) A((void**)&z->ls, rows * z->wb * C64 * sizeof(__half));
    A((void**)&z->li, rows * C64 * sizeof(__half));
    A((void**)&z->rexp, sizeof(int) * z->M128);
    A((void**)&z->lexp, sizeof(int) * z->M128);
    A((void**)&z->wexp, sizeof(int) * z->nbc);
    A((void**)&z->flags, sizeof(int) * chol64_flags(z));
    if (!z->own_ls) A((void**)&z->diag, sizeof(double) * z->M128);
    if (e == cudaSuccess) e = cudaFuncSetAttribute(k_chol64, cudaFuncAttributeMaxDynamicSharedMemorySize, oz_smem(CS));
    if (e == cudaSuccess)
        e = cudaFuncSetAttribute(k_chol64_plain, cudaFuncAttributeMaxDynamicSharedMemorySize, CP_SMEM);
    int rc = QLP_OK;
    if (e != cudaSuccess) {
        cudaGetLastError();
        set_error("%s (%d)", "FP64 factorisation workspace", (int)e);
        rc = (e == cudaErrorMemoryAllocation) ? QLP_ERR_NOMEM : QLP_ERR_CUDA;
    } else if (make_map_box(&z->ls_a, z->ls, rows, z->wb * C64, true, OZ_TM, OZ_KS) != QLP_OK ||
               make_map_box(&z->ls_b, z->ls, rows, z->wb * C64, true, OZ_TN, OZ_KS) != QLP_OK ||
               make_map_box(&z->li_b, z->li, rows, C64, true, OZ_TN, OZ_KS) != QLP_OK) {
        set_error("%s (%d)", "cuTensorMapEncodeTiled unavailable or failed", 0);
        rc = QLP_ERR_CUDA;
    }
    if (rc != QLP_OK) { chol64_free(z); return rc; }
    *out = z;
    return QLP_OK;
}

// The flags of a factorisation and of one pair of solves.
void chol64_clear(const Chol64Work* z, ClearList& l)
{
    l.add(z->flags, sizeof(int) * chol64_flags(z));
}

// which: 0 F, 1 R (the not-SPD flag).  half_width: how far below the diagonal
// the matrix reaches (R: two grid rows), or past M.  ctas: the grid's size.
void launch_cholesky_fp64(double* A, int ld, int M_max, GridState* gs, int which, int half_width, int ctas,
                          Chol64Work* z, double* linv, cudaStream_t st)
{
    const int nb = (M_max + C64 - 1) / C64;
    const int band = chol64_band(half_width, M_max);
    const int tiles = nb * std::min((nb + 1) / 2, band / 2 + 1);
    k_chol64_prep<<<(M_max + 255) / 256, 256, 0, st>>>(gs, A, ld, z->rexp);
    int* redo = z->diag ? z->flags + chol64_flags(z) - 2 : nullptr;
    k_chol64<<<std::max(1, std::min(tiles, ctas)), OZ_THREADS, oz_smem(CS), st>>>(
        z->ls_a, z->ls_b, z->li_b, gs, A, ld, which, band, z->M128, z->nbc, z->wb, z->ls, z->li, z->rexp, z->lexp, z->wexp,
        z->flags, linv, redo, z->diag);
    count_launches(2);
    if (!redo) return;
    k_chol64_plain<<<std::max(1, std::min(nb * (nb + 1) / 2, ctas)), 256, CP_SMEM, st>>>(gs, A, ld, z->diag, z->nbc,
                                                                                    z->flags, redo, redo + 1, linv);
    count_launches(1);
}

void launch_solve_fp64(Work& w, int M_max, cudaStream_t st)
{
    Chol64Work* z = w.cholF;
    const int nb = (M_max + C64 - 1) / C64;
    int* flags = z->flags + (size_t)z->nbc * z->nbc + z->nbc + 1;
    k_trsv64_fwd<<<nb, 256, 0, st>>>(w.F, w.ldF, w.linv, w.gs, w.D, w.tmp, flags);
    k_trsv64_bwd<<<nb, 256, 0, st>>>(w.F, w.ldF, w.linv, w.gs, w.tmp, w.s, flags + z->nbc);
    count_launches(2);
}

}  // namespace qlpix
