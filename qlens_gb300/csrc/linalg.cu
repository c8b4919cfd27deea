// linalg.cu -- FP64 dense algebra of the inversion:
//   D = L'^T C^-1 d, curvature R and F += lambda R, log det, the
//   model image, chi^2, s^T R s and the final -2 log(evidence).
// Reference: QLens::create_lensing_matrices_from_Lmatrix_dense
// (pixelgrid.cpp:15590-15736), add_regularization_term_to_dense_Fmatrix
// (15781-15819), invert_lens_mapping_dense (17346-17396), Cholesky_dcmp_packed
// (17071-17105), Cholesky_solve_lower_packed (17230-17246),
// Cholesky_logdet_lower_packed (17201-17210), Rmatrix_determinant_dense
// (18176-18191), calculate_image_pixel_surface_brightness_dense (18268-18290),
// calculate_regularization_prior_term (15821-15863), chi^2 and evidence
// assembly (lens.cpp:12950-13016, 12608-12615).
//
// Matrices are dense row-major with leading dimension ldF; the lower triangle
// holds F (and later its Cholesky factor).  Sizes past the active count M are
// padded to a multiple of 64 with an identity block, which leaves log det and
// the solution unchanged.  Every kernel reads N and M from the device-side
// GridState, so the launch sequence never waits for the host.
#include "qlpix_ctx.h"
#include "chol.cuh"

namespace qlpix {

#define NB 64

__device__ __forceinline__ int mpad64(int M) { return (M + 63) & ~63; }

// ---- a graph replay's parameters and result, from and to pinned host memory ----
__global__ void k_job_in(const Job* jobs, unsigned ring, const unsigned* count, EvalParams* ep, int trial)
{
    const EvalParams* src = jobs[*count & (ring - 1)].ep;
    if (trial) {
        if (threadIdx.x == 0) ep->regparam = src->regparam;
        return;
    }
    const unsigned long long* s = reinterpret_cast<const unsigned long long*>(src);
    unsigned long long* d = reinterpret_cast<unsigned long long*>(ep);
    for (int i = threadIdx.x; i < (int)(sizeof(EvalParams) / 8); i += blockDim.x) d[i] = s[i];
}

__global__ void k_job_out(const Job* jobs, unsigned ring, unsigned* count, const EvalOut* out)
{
    static_assert(sizeof(EvalParams) % 8 == 0 && sizeof(EvalOut) % 8 == 0, "copied as 8-byte words");
    const unsigned q = *count;
    EvalOut* dst = jobs[q & (ring - 1)].out;
    if (dst)
        for (int i = threadIdx.x; i < (int)(sizeof(EvalOut) / 8); i += blockDim.x)
            reinterpret_cast<unsigned long long*>(dst)[i] = reinterpret_cast<const unsigned long long*>(out)[i];
    __syncthreads();
    if (threadIdx.x == 0) *count = q + 1;
}

void launch_job_in(const Job* jobs, unsigned ring, unsigned* count, EvalParams* ep, bool trial, cudaStream_t st)
{
    k_job_in<<<1, 256, 0, st>>>(jobs, ring, count, ep, trial ? 1 : 0);
    count_launches(1);
}

void launch_job_out(const Job* jobs, unsigned ring, unsigned* count, const EvalOut* out, cudaStream_t st)
{
    k_job_out<<<1, 32, 0, st>>>(jobs, ring, count, out);
    count_launches(1);
}

// ---- clearing and copying ----
__global__ void __launch_bounds__(256) k_clear(ClearList l)
{
    for (int k = 0; k < l.n; k++) {
        const ClearItem it = l.item[k];
        const uint4 v = make_uint4(it.value, it.value, it.value, it.value);
        uint4* p4 = reinterpret_cast<uint4*>(it.p);
        const unsigned n4 = ((size_t)it.p & 15) == 0 ? it.words / 4 : 0;
        for (unsigned i = blockIdx.x * blockDim.x + threadIdx.x; i < n4; i += gridDim.x * blockDim.x) p4[i] = v;
        unsigned* p = reinterpret_cast<unsigned*>(it.p);
        for (unsigned i = 4 * n4 + blockIdx.x * blockDim.x + threadIdx.x; i < it.words; i += gridDim.x * blockDim.x)
            p[i] = it.value;
    }
}

int launch_clear(const ClearList& l, cudaStream_t st)
{
    if (l.full) {
        set_error("%s (%d)", "too many buffers to clear", l.n);
        return QLP_ERR_ARG;
    }
    size_t words = 0;
    for (int k = 0; k < l.n; k++) words += l.item[k].words;
    const int blocks = (int)((words / 4 + 1023) / 1024);
    k_clear<<<blocks < 1 ? 1 : (blocks > 152 * 2 ? 152 * 2 : blocks), 256, 0, st>>>(l);
    count_launches(1);
    return QLP_OK;
}

__global__ void __launch_bounds__(256) k_clear_band(char* __restrict__ A, size_t ld_bytes, int esize, int blk, int back,
                                                    const GridState* __restrict__ gs)
{
    const int row = blockIdx.x * 8 + (threadIdx.x >> 5), i = row / blk;
    if (row >= (gs->M + blk - 1) / blk * blk) return;
    const int c0 = blk * max(0, i - back), c1 = blk * (i + 1);
    uint4* p = reinterpret_cast<uint4*>(A + row * ld_bytes + (size_t)c0 * esize);
    for (int k = threadIdx.x & 31; k < (c1 - c0) * esize / 16; k += 32) p[k] = make_uint4(0u, 0u, 0u, 0u);
}

void launch_clear_band(void* A, int ld, int esize, int rows, int blk, int back, const GridState* gs, cudaStream_t st)
{
    k_clear_band<<<(rows + 7) / 8, 256, 0, st>>>((char*)A, (size_t)ld * esize, esize, blk, back, gs);
    count_launches(1);
}

__global__ void __launch_bounds__(256) k_copy_square(char* __restrict__ dst, const char* __restrict__ src,
                                                     size_t ld_bytes, int esize, int blk,
                                                     const GridState* __restrict__ gs)
{
    const int Mp = (gs->M + blk - 1) / blk * blk, row = blockIdx.x;
    if (row >= Mp) return;
    const uint4* s = reinterpret_cast<const uint4*>(src + row * ld_bytes);
    uint4* d = reinterpret_cast<uint4*>(dst + row * ld_bytes);
    // the lower triangle, in whole blocks
    const int n = blk * (row / blk + 1) * esize / 16;
    for (int k = threadIdx.x; k < n; k += blockDim.x) d[k] = s[k];
}

void launch_copy_square(void* dst, const void* src, int ld, int esize, int blk, const GridState* gs, int rows,
                        cudaStream_t st)
{
    k_copy_square<<<rows, 256, 0, st>>>((char*)dst, (const char*)src, (size_t)ld * esize, esize, blk, gs);
    count_launches(1);
}

// ---- D = L'^T (C^-1 d) ----
// Eight cells a CTA over the live 32-pixel stages of their 64-cell block: a warp
// takes every eighth stage, its lanes the stage's pixels, all eight cells beside
// each other (C^-1 d is formed once for them); then a shuffle tree and the warps in
// order.  The FP64 pipe bounds it (one multiply-add a live entry; skipping the zeros
// among them by a test cost more than they).  Two multiplies and an add for every
// entry of a row-wise L' before: 2,934 cells x 11,772 pixels 194 -> 72 us, and the
// model image likewise 76 -> 54 us.
#define D_CELLS 8
__global__ void __launch_bounds__(256) k_D(const GridState* __restrict__ gs, const double* __restrict__ L, int ldL,
                                           const unsigned char* __restrict__ nz, int nst,
                                           const double* __restrict__ dvec, const double* __restrict__ cvec,
                                           double* __restrict__ D)
{
    __shared__ double part[8][D_CELLS];
    const int N = gs->N, M = gs->M;
    const int c0 = blockIdx.x * D_CELLS, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    if (c0 >= mpad64(M)) return;
    double acc[D_CELLS];
    #pragma unroll
    for (int k = 0; k < D_CELLS; k++) acc[k] = 0;
    if (c0 < M) {
        const unsigned char* live = nz + (size_t)(c0 / 64) * nst;
        for (int st = warp; st * 32 < N; st += 8) {
            const int r = st * 32 + lane;
            if (!live[st] || r >= N) continue;
            const double w = dvec[r] * cvec[r];
            #pragma unroll
            for (int k = 0; k < D_CELLS; k++)
                if (c0 + k < M) acc[k] = fma(L[(size_t)(c0 + k) * ldL + r], w, acc[k]);
        }
    }
    #pragma unroll
    for (int k = 0; k < D_CELLS; k++) {
        for (int o = 16; o > 0; o >>= 1) acc[k] += __shfl_xor_sync(0xffffffffu, acc[k], o);
        if (lane == 0) part[warp][k] = acc[k];
    }
    __syncthreads();
    if (threadIdx.x < D_CELLS) {
        double a = 0;
        for (int k = 0; k < 8; k++) a += part[k][threadIdx.x];
        D[c0 + threadIdx.x] = a;
    }
}

void launch_D(Work& w, int M_max, cudaStream_t st)
{
    k_D<<<(M_max + 63) / 64 * (64 / D_CELLS), 256, 0, st>>>(w.gs, w.Lpsf, w.ldL, oz_nz(w.oz), oz_nst(w.oz),
                                                                 w.dvec, w.cvec, w.D);
    count_launches(1);
}

// ---- curvature R (dense lower) and F += lambda R ----
// R = Hx^T Hx + Hy^T Hy with Hx rows (-2 at a, +1 at active x-neighbours) and
// Hy likewise (SourcePixel::generate_hmatrices, pixelgrid.cpp:2968-3071;
// generate_Rmatrix_from_hmatrices 3073-3240).  In closed form per active cell:
// diagonal 8 + #active 4-neighbours, -4 for an active +-1 neighbour, +1 for an
// active +-2 neighbour whose middle cell is active.
__device__ __forceinline__ int act_at(const int* ai, int snx, int sny, int i, int j)
{
    if (i < 0 || j < 0 || i >= snx || j >= sny) return -1;
    return ai[j * snx + i];
}

__global__ void k_reg(const GridState* __restrict__ gs, const int* __restrict__ ai,
                      const double* __restrict__ regp, double* __restrict__ F, double* __restrict__ R, int ldF,
                      int do_reg, int parts)
{
    const bool toF = parts & REG_F, toR = parts & REG_R;
    const double regparam = *regp;
    const int snx = gs->snx, sny = gs->sny;
    const int M = gs->M, Mp = mpad64(M);
    const int ncell = snx * sny;
    for (int c = blockIdx.x * blockDim.x + threadIdx.x; c < ncell + (Mp - M); c += gridDim.x * blockDim.x) {
        if (c >= ncell) {   // identity padding
            int i = M + (c - ncell);
            if (toF) F[(size_t)i * ldF + i] = 1.0;
            if (do_reg && toR) R[(size_t)i * ldF + i] = 1.0;
            continue;
        }
        if (!do_reg) continue;
        const int a = ai[c];
        if (a < 0) continue;
        const int ci = c % snx, cj = c / snx;
        int nb1[4] = {act_at(ai, snx, sny, ci + 1, cj), act_at(ai, snx, sny, ci - 1, cj),
                      act_at(ai, snx, sny, ci, cj + 1), act_at(ai, snx, sny, ci, cj - 1)};
        int nb2[4] = {act_at(ai, snx, sny, ci + 2, cj), act_at(ai, snx, sny, ci - 2, cj),
                      act_at(ai, snx, sny, ci, cj + 2), act_at(ai, snx, sny, ci, cj - 2)};
        double diag = 8.0;
        for (int k = 0; k < 4; k++) if (nb1[k] >= 0) diag += 1.0;
        if (toR) R[(size_t)a * ldF + a] = diag;
        if (toF) F[(size_t)a * ldF + a] += regparam * diag;
        for (int k = 0; k < 4; k++) {
            int b = nb1[k];
            if (b >= 0 && b < a) {
                if (toR) R[(size_t)a * ldF + b] = -4.0;
                if (toF) F[(size_t)a * ldF + b] += regparam * -4.0;
            }
            int b2 = nb2[k];
            if (b2 >= 0 && nb1[k] >= 0 && b2 < a) {
                if (toR) R[(size_t)a * ldF + b2] = 1.0;
                if (toF) F[(size_t)a * ldF + b2] += regparam * 1.0;
            }
        }
    }
}

void launch_regularization(const SrcOpts& so, Work& w, int M_max, const double* regp, int parts, cudaStream_t st)
{
    const int ncell = so.snx * so.sny;
    int total = ncell + 64;
    k_reg<<<(total + 255) / 256, 256, 0, st>>>(w.gs, w.active_index, regp, w.F, w.R, w.ldF, so.regularization,
                                               parts);
    count_launches(1);
    (void)M_max;
}

// ---- log det of a factor (the factorisations and solves: cholfp64.cu) ----
void launch_logdet_R(const double* A, int ld, Work& w, cudaStream_t st)
{
    k_logdet_t<double><<<1, 1024, 0, st>>>(A, ld, w.gs, w.out);
    count_launches(1);
}

// ---- model image, chi^2, s^T R s and the evidence ----
// 32 pixels a CTA, a lane each; a warp takes eight cells of every live 64-cell
// block, then the warps' sums in order.
__global__ void __launch_bounds__(256) k_model(const GridState* __restrict__ gs, const double* __restrict__ L,
                                               int ldL, const unsigned char* __restrict__ nz, int nst,
                                               const double* __restrict__ s, double* __restrict__ model)
{
    __shared__ double part[8][32];
    const int N = gs->N, M = gs->M;
    const int st = blockIdx.x, lane = threadIdx.x & 31, warp = threadIdx.x >> 5, r = st * 32 + lane;
    if (st * 32 >= N) return;
    double acc = 0;
    for (int cb = 0; cb * 64 < M; cb++) {
        if (!nz[(size_t)cb * nst + st]) continue;
        const int c0 = cb * 64 + warp * 8;
        const double* p = L + (size_t)c0 * ldL + r;
        double v[8];
        #pragma unroll
        for (int k = 0; k < 8; k++) v[k] = (c0 + k < M && r < N) ? p[(size_t)k * ldL] : 0.0;
        #pragma unroll
        for (int k = 0; k < 8; k++)
            if (c0 + k < M) acc = fma(v[k], s[c0 + k], acc);
    }
    part[warp][lane] = acc;
    __syncthreads();
    if (warp == 0 && r < N) {
        double a = 0;
        for (int k = 0; k < 8; k++) a += part[k][lane];
        model[r] = a;
    }
}

// chi^2, s^T R s, log det F from the factor A's diagonal, and the evidence: FINAL_CTAS
// CTAs sum their shares, and the last of them adds those in a fixed order and puts
// the result together.  The FP64 pipe bounds the sums (logarithms, the stencil of R):
// one CTA for each of log det and the rest took 30 + 45 us at 2,934 cells and 11,772
// pixels, now 17 us together.
#define FINAL_CTAS 32
#define FINAL_SUMS 5
__global__ void __launch_bounds__(256) k_final(StaticData sd_, SrcOpts so_, const GridState* __restrict__ gs,
                                               const int* __restrict__ rowidx, const double* __restrict__ model,
                                               const double* __restrict__ s, const int* __restrict__ ai,
                                               const double* __restrict__ regp, const void* __restrict__ A, int ld,
                                               int fp32, double* __restrict__ part, int* __restrict__ count,
                                               EvalOut* out)
{
    const StaticData sd = eval_shape(sd_);
    const SrcOpts so = eval_grid(so_, sd_);
    const double regparam = *regp;
    __shared__ double red[FINAL_SUMS][8];
    __shared__ int last;
    const int M = gs->M;
    const int first = blockIdx.x * blockDim.x + threadIdx.x, stride = gridDim.x * blockDim.x;
    double chi = 0, es = 0, chi_act = 0, logc = 0, logd = 0;
    for (int m = first; m < sd.n_mask; m += stride) {
        const int pix = sd.mpix[m];
        const double c = sd.use_noise_map ? sd.covinv[pix] : sd.cov_inverse;
        const int r = rowidx[m];
        double dd = (r >= 0) ? model[r] - sd.data[pix] : sd.data[pix];
        chi += dd * dd * c;
        if (r >= 0) chi_act += dd * dd * c;     // the pixels the lambda optimisation's chi^2 runs over
        if (r >= 0 && sd.noise_term && sd.use_noise_map) logc += log(c);
    }
    if (so.regularization && regparam != 0) {
        const int snx = so.snx, sny = so.sny;
        for (int cidx = first; cidx < snx * sny; cidx += stride) {
            const int a = ai[cidx];
            if (a < 0) continue;
            const int ci = cidx % snx, cj = cidx / snx;
            int nb1[4] = {act_at(ai, snx, sny, ci + 1, cj), act_at(ai, snx, sny, ci - 1, cj),
                          act_at(ai, snx, sny, ci, cj + 1), act_at(ai, snx, sny, ci, cj - 1)};
            int nb2[4] = {act_at(ai, snx, sny, ci + 2, cj), act_at(ai, snx, sny, ci - 2, cj),
                          act_at(ai, snx, sny, ci, cj + 2), act_at(ai, snx, sny, ci, cj - 2)};
            double diag = 8.0, rs = 0;
            for (int k = 0; k < 4; k++) {
                if (nb1[k] >= 0) { diag += 1.0; rs += -4.0 * s[nb1[k]]; }
                if (nb2[k] >= 0 && nb1[k] >= 0) rs += s[nb2[k]];
            }
            rs += diag * s[a];
            es += s[a] * rs;
        }
    }
    for (int i = first; i < M; i += stride) {
        const size_t d = (size_t)i * ld + i;
        logd += log(fabs(fp32 ? (double)reinterpret_cast<const float*>(A)[d] : reinterpret_cast<const double*>(A)[d]));
    }
    double sum[FINAL_SUMS] = {chi, es, chi_act, logc, logd};
    #pragma unroll
    for (int k = 0; k < FINAL_SUMS; k++) {
        for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
        if ((threadIdx.x & 31) == 0) red[k][threadIdx.x >> 5] = sum[k];
    }
    __syncthreads();
    if (threadIdx.x < FINAL_SUMS) {
        double t = 0;
        for (int k = 0; k < 8; k++) t += red[threadIdx.x][k];
        part[threadIdx.x * FINAL_CTAS + blockIdx.x] = t;
        __threadfence();
    }
    __syncthreads();
    if (threadIdx.x == 0) last = atomicAdd(count, 1) == (int)gridDim.x - 1;
    __syncthreads();
    if (!last || threadIdx.x >= 32) return;
    __threadfence();
    #pragma unroll
    for (int k = 0; k < FINAL_SUMS; k++) {
        sum[k] = __ldcg(part + k * FINAL_CTAS + threadIdx.x);
        for (int o = 16; o > 0; o >>= 1) sum[k] += __shfl_xor_sync(0xffffffffu, sum[k], o);
    }
    if (threadIdx.x == 0) {
        *count = 0;                                       // for the next evaluation
        const double c2 = sum[0], e2 = sum[1], ca = sum[2], lc = sum[3];
        out->logdet_F = 2 * sum[4];
        double regterms = 0, loglike = 0;
        if (so.regularization && M > 0) {
            if (regparam != 0) {
                regterms = regparam * e2 - M * log(regparam) - out->logdet_R;
                loglike += regterms;
            }
            loglike += out->logdet_F;
        }
        loglike += c2;
        // the pixel-noise normalisation, QLens 'include_noise_term_in_loglike'
        // (lens.cpp:13033-13043): minus the log of C^-1 over the active pixels
        // with a noise map, or the masked-pixel count times log(1/sigma^2)
        // without one, plus the masked-pixel count times log(2 pi)
        if (sd.noise_term) {
            loglike -= sd.use_noise_map ? lc : sd.n_mask * log(sd.cov_inverse);
            loglike += sd.n_mask * log(6.28318530717958647692);
        }
        int status = gs->status;
        if (status == 0 && (gs->not_spd_F || gs->not_spd_R)) status = QLP_ERR_NOT_SPD;
        // QLens::chisq_regparam_dense (pixelgrid.cpp:16688-16692): Ed + prior + log det F
        out->f_regopt = ca + ((so.regularization && M > 0) ? ((regparam != 0 ? regterms : 0.0) + out->logdet_F) : 0.0);
        out->chisq0 = c2;
        out->Es_times_two = e2;
        out->regterms = regterms;
        out->m2logev = (status == QLP_ERR_NO_SOURCE_PIXELS) ? 2e30 : loglike;
        out->n_active_pixels = gs->N;
        out->n_active_src = M;
        out->L_nnz = gs->nnz;
        out->status = status;
    }
}

void launch_model_chi2(const StaticData& sd, const SrcOpts& so, Work& w, int N_max, const double* regp,
                       const void* factor, int ld, bool mixed, cudaStream_t st)
{
    if (N_max > 0 && !mixed) {
        k_model<<<(N_max + 31) / 32, 256, 0, st>>>(w.gs, w.Lpsf, w.ldL, oz_nz(w.oz), oz_nst(w.oz), w.s, w.model);
        count_launches(1);
    }
    k_final<<<FINAL_CTAS, 256, 0, st>>>(sd, so, w.gs, w.rowidx, w.model, w.s, w.active_index, regp, factor, ld,
                                        mixed ? 1 : 0, w.fpart, w.fcount, w.out);
    count_launches(1);
}

}  // namespace qlpix
