// qlpix_ctx.h -- the context object behind qlp_ctx* (host runtime).
#pragma once
#include <cuda_runtime.h>
#include <string>
#include <utility>
#include <vector>
#include "qlpix_internal.h"

#define QLP_N_STAGES 6
#define QLP_MAX_SLOTS 64
#define QLP_LOADS 3                 // alone, a few evaluations in flight, many (load_of)
#define QLP_JOB_RING 1024           // graph replays queued per slot (a power of two: the device's count wraps)

namespace qlpix {

// The launch sequence captured as a CUDA graph, sized for the slot's capacity
// (any mask and source grid that fit), valid for one (precision, capacity, NFW,
// NFW mode, lambda optimisation) combination and graph generation; with the
// lambda optimisation on there is one for the lambda-independent part and one
// for a lambda trial.
struct SlotGraph {
    cudaGraphExec_t exec = nullptr;
    int key[7] = {0, 0, 0, 0, 0, 0, 0};
    long long gen = 0;
    long long launches = 0;         // kernels per replay
};

// One evaluation lane: a stream and the full per-evaluation workspace.  A
// batch spreads its instances over several slots so that the sequential
// parts of one evaluation (Cholesky pivots, triangular solves) overlap the
// parallel parts of others.
struct Slot {
    cudaStream_t stream = nullptr;
    Work w{};
    void* mixed = nullptr;          // mixed-precision workspace (mixed.cu)
    int M_cap = 0;                  // capacity in source cells (multiple of 64)
    int N_cap = 0;                  // capacity in masked pixels
    int nsub_cap = 0;
    int snx_cap = 0, sny_cap = 0;
    int npix_pad = 0;               // image pixels with a PSF-half-width border: (nx + 2 (pnx/2)) (ny + 2 (pny/2))
    int img_nx = 0, img_ny = 0;     // image and PSF sizes (the PSF-to-X band layout)
    int psf_nx = 0, psf_ny = 0;
    bool fp64_mats = false;         // F and R in FP64 allocated
    cudaEvent_t done = nullptr;
    // second stream of the slot: R's factorisation runs beside F's
    cudaStream_t side = nullptr;
    cudaEvent_t side_fork = nullptr, side_join = nullptr;
    SlotGraph graphs[2][QLP_LOADS];     // [a lambda trial's][load_of]
    // what the graph's replays work on: replay number q takes entry q % QLP_JOB_RING
    // of the ring (pinned); the device counts the replays that are done
    Job* jobs = nullptr;
    unsigned* job_count = nullptr;
    unsigned long long job_no = 0;      // replays launched
    unsigned long long job_synced = 0;  // ... at the stream's last synchronisation for the ring
    OsbWork osb{};                  // outside-surface-brightness pass (allocated when the prior is on)
    int osb_nsub = 0;               // its capacity in sub-pixels
};

}  // namespace qlpix

struct qlp_ctx {
    int device = 0;
    cudaStream_t own_stream = nullptr;
    cudaStream_t stream = nullptr;
    int precision = QLP_FP64;
    int max_slots = 16;                   // schedule: evaluations in flight
    int ray_threads = 256;                // schedule: ray-shooting CTA size
    int psfx_threads = 256;               // schedule: k_psf_x CTA size
    int psfx_split = 1;                   // schedule: accepted and reported, without effect, as psfx_mode
    int psfx_mode = -1;                   // (-1: set from the PSF size at creation)

    // lens model
    std::vector<qlp_lens> lenses;
    std::vector<qlp_fit_param> fit;    // qlp_set_fit_params
    qlp_planes planes{};

    // host copies of the static inputs
    int nx = 0, ny = 0;
    std::vector<int> mpix;                // masked pixels of the image mask (j-outer, i-inner)
    qlp_srcgrid_opts opts{};

    // device copies
    double* d_xvals = nullptr;
    double* d_yvals = nullptr;
    double* d_data = nullptr;
    double* d_covinv = nullptr;
    double* d_psf = nullptr;
    int2* d_psf_fine = nullptr;    // the plain path's (StaticData::psf_fine)
    int psf_bits = 0;              // half a unit of its taps is at most 2^-psf_bits of the largest (0: not fixed)
    std::vector<double> covinv;    // noise map: C^-1 per pixel
    int* d_psf_int = nullptr;      // the PSF on the PSF-to-X fixed-point grid (StaticData::psf_int)
    int* d_mpix = nullptr;

    // extra masks for batched evaluation (device mpix lists, concatenated)
    std::vector<int> mask_off, mask_cnt;
    int* d_inst_mpix = nullptr;

    qlpix::StaticData sd{};
    qlpix::SrcOpts so{};
    std::vector<qlpix::Slot> slots;       // slots[0] serves qlp_eval

    qlpix::EvalOut* h_out = nullptr;      // pinned, one per batch instance
    int h_out_cap = 0;
    qlpix::EvalOut* h_trial = nullptr;    // pinned, one per slot: results of lambda trials
    qlpix::Job* jobs = nullptr;           // pinned: the slots' rings of jobs
    unsigned* job_counts = nullptr;       // device: replays run, one per slot
    std::vector<double> regopt_lam;       // per batch instance: the lambda of its result
    std::vector<int> regopt_evals;        // per batch instance: lambda trials run
    cudaEvent_t ev[QLP_N_STAGES + 1] = {};
    cudaEvent_t fork = nullptr, join = nullptr;
    std::vector<cudaEvent_t> ev_pool;     // (QLP_N_STAGES+1) per batched instance
    qlpix::EvalParams* h_ep = nullptr;    // pinned, one per batch instance
    int h_ep_cap = 0;
    int in_flight = 1;                    // evaluations in flight in the current call
    int use_graphs = 1;                   // batched evaluation replays captured graphs
    int refine = 1;                       // FP64 refinement sweeps of the mixed path's amplitudes
    // regularisation-parameter optimisation (QLens 'optimize_regparam on'):
    // Brent's method over log10(lambda), QLens's defaults
    int regopt = 0;
    double regopt_minlog = -3.0, regopt_maxlog = 5.0, regopt_tol = 0.01;
    int regopt_maxit = 20;
    int nfw_mode = QLP_NFW_QUADRATURE;    // NFW deflection: quadrature or trained surrogate
    double nfw_threshold = 2e-5;          // surrogate error bound (arcsec) above which a ray falls back
    double nfw_tol = 1e-3;                // the NFW quadrature's tolerance (QLens integral_tolerance)
    // outside-surface-brightness prior (QLens 'outside_sb_prior'): settings,
    // device tables of the extended mask, background noise of the image
    int osb_on = 0;
    qlpix::OsbStatic osb{};
    unsigned char* d_emask = nullptr;
    unsigned char* d_inmask = nullptr;
    int* d_epix = nullptr;
    int* d_eoff = nullptr;
    double bg_noise = 0;
    long long graph_gen = 1;              // bumped whenever captured graphs go stale
    long long last_h2d = 0, last_d2h = 0; // bytes moved by the last call
    float stage_ms[QLP_N_STAGES] = {};
    float device_ms = 0;
    long long last_launches = 0;
};

namespace qlpix {
int ctx_init(qlp_ctx* c, const qlp_image* im, const qlp_psf* psf, const qlp_srcgrid_opts* opts);
void ctx_free(qlp_ctx* c);
int ctx_eval(qlp_ctx* c, const double* lens_params, double regparam, qlp_result* out);
int ctx_set_masks(qlp_ctx* c, const unsigned char* masks, int n_masks);
int ctx_eval_batch(qlp_ctx* c, const double* params, const double* regparams, const qlp_instance* inst, int n,
                   qlp_result* out);
int ctx_dump(qlp_ctx* c, double* srcpt_xy, int* L_rowptr, int* L_index, double* L_value, int* active_index,
             double* D, double* s, double* model);
int ctx_dump_Lpsf(qlp_ctx* c, int rows, double* out);
int factor_ctas(const qlp_ctx* c, int nb);
int make_lens_rec(LensRec& L, const qlp_lens& d, const double* p);
int fit_set(qlp_ctx* c, const qlp_fit_param* fp, int n);
int fit_loglike_batch(qlp_ctx* c, const double* x, int n, double* loglike, qlp_result* out);
int fit_terms(const qlp_fit_param* fp, int n, const double* x, double* t, int* penalised, double* terms);
bool is_nfw_type(int type);
int n_params_of(int type);
void set_error(const char* fmt, const char* a, int code);
// mixed.cu
int mixed_init(Slot& slot);
void mixed_free(Slot& slot);
// Buffers that live and die together, in one device allocation (an allocation each,
// some 70 a slot, was a third of a batch's first pass).
struct Arena {
    std::vector<std::pair<void**, size_t>> parts;          // where each part's address goes, its offset
    size_t bytes = 0;
    template <typename T>
    void add(T** p, size_t n)
    {
        parts.emplace_back(reinterpret_cast<void**>(p), bytes);
        bytes += (sizeof(T) * (n > 0 ? n : 1) + 511) / 512 * 512;
    }
    cudaError_t commit(void** base) const
    {
        const cudaError_t e = cudaMalloc(base, bytes);
        for (size_t k = 0; e == cudaSuccess && k < parts.size(); k++)
            *parts[k].first = static_cast<char*>(*base) + parts[k].second;
        return e;
    }
};
void csc_layout(Csc& o, const Slot& c, int M_cap, bool fine, Arena& ar);
// launch sequences of one evaluation: the whole of it, or, for the
// regularisation-parameter optimisation, its lambda-independent part and one
// lambda trial
#define PIPE_ALL 0
#define PIPE_PRE 1
#define PIPE_TRIAL 2
int mixed_ensure_f0(Slot& slot);
const float* mixed_factor(Slot& slot, int& ld);
void mixed_clear(Slot& slot, ClearList& l, bool trial);
int run_inversion_mixed(const qlp_ctx* c, Slot& slot, const StaticData& sd, const SrcOpts& so, const double* regp,
                        int part, cudaStream_t st,
                        cudaEvent_t* ev);
// autotune.cpp
int ctx_get_schedule(const qlp_ctx* c, qlp_schedule* out);
// outside.cu / ctx.cpp: the outside-surface-brightness prior
int ctx_set_outside_sb(qlp_ctx* c, int on, double frac, double noise_frac, const unsigned char* emask, int ens);
int ctx_set_schedule(qlp_ctx* c, const qlp_schedule* s);
int ctx_autotune(qlp_ctx* c, const double* params, const double* lambdas, const qlp_instance* inst, int n, int reps,
                 qlp_tune_report* rep);
void ctx_trim_slots(qlp_ctx* c, int keep);
// surrogate.cu
int surrogate_train(int device, const qlp_surrogate_opts* o, qlp_surrogate_report* rep);
bool surrogate_ready(int device);
int surrogate_grad_check(int device, const float* params, const float* x, const float* t, int batch, double* loss,
                         float* grad);
int surrogate_eval(int device, const double* rpq, int n, double* t_net, double* G_quad, double* B, double* bound);
int launch_raytrace_sur(const StaticData& sd, Work& w, double thresh, int defer_lens, cudaStream_t st);
int launch_surrogate_exact(const StaticData& sd, const SrcOpts& so, Work& w, double eps_g, int step,
                           cudaStream_t st);
}  // namespace qlpix
