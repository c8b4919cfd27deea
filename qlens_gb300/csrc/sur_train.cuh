// sur_train.cuh -- training step of the learned NFW deflection's network
// (3 -> 128 -> 128 -> 128 -> 128 -> 2, tanh), FP32 on the CUDA cores.
//
// Three launches a step, each output one FMA chain in ascending order:
//   k_sur_chain   16 RT rows of the batch per CTA through the whole network and
//                 back: activations and their gradients stay in shared memory
//                 between layers (and are stored for the weight gradients), the
//                 next layer's weights are copied in while a layer runs, and a
//                 thread holds an RT x 8 block of outputs in registers;
//   k_sur_wgrad   the weight gradients of all layers, split over the batch into
//                 chains of 256 to 511 rows (64 x 128 tiles), and the bias
//                 gradients' sums over every 256th row;
//   k_sur_update  the splits summed in order, Adam, and the transposed weights
//                 that k_sur_chain's way back reads.
// Bound by the FP32 pipe (4.9 GFLOP a step of 16,384 rows, 63 us at the peak of
// 128 FMA a clock and SM).  One strided GEMM per layer and direction, 64x64 tiles
// of single-word loads without overlap and ten small reductions, took 0.63 ms a
// step; 0.13 now (chain 0.073, weight gradients 0.049, update 0.010).
#pragma once

namespace qlpix {

struct SurTrain {
    int bs, KS, ksplit;       // batch rows; weight-gradient splits and their rows
    const float *x, *t, *w;   // inputs [bs][3], targets [bs][2], loss weights or null
    float* P;                 // parameters
    float* PT;                // the three 128 x 128 layers transposed
    float *m1, *m2, *grad;
    float* act;               // [6][bs][128]: 1..4 the hidden layers' outputs, 5 the output [bs][2]
    float* dz;                // [4][bs][128] gradients at the layers' sums, then [bs][2] at the output
    float* gpart;             // [3][KS][128][128], [KS][3][128], [KS][128][2]
    float* cpart;             // [4][256][128], [256][2]
    double* lpart;
};

#define ST_HH (SUR_H * SUR_H)
#define ST_THREADS 256
#define ST_CHAIN_SMEM ((3 * ST_HH + 2 * SUR_H + 2 * SUR_H) * 4)
#define ST_WG_K 32                                            // samples a stage
#define ST_WG_STAGE (ST_WG_K * (64 + SUR_H))                  // floats
#define ST_WG_SMEM (3 * ST_WG_STAGE * 4)

static inline size_t st_gpart_floats(int KS) { return (size_t)KS * (3 * ST_HH + 5 * SUR_H); }
#define ST_CPART_FLOATS (4 * 256 * SUR_H + 512)

__device__ __forceinline__ void st_cp16(float* dst, const float* src, bool valid)
{
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;" ::"r"(smem_u32(dst)), "l"(src), "r"(valid ? 16 : 0)
                 : "memory");
}
__device__ __forceinline__ void st_commit() { asm volatile("cp.async.commit_group;" ::: "memory"); }
template <int N>
__device__ __forceinline__ void st_wait() { asm volatile("cp.async.wait_group %0;" ::"n"(N) : "memory"); }

// acc[v..v+1] += a (x[v], x[v+1]) for 8 columns: two FMAs an instruction, the same
// roundings (the issue slots, not only the pipe, bound a loop of single ones)
__device__ __forceinline__ void st_fma8(float a, const float (&x)[8], float (&acc)[8])
{
    unsigned long long aa;
    asm("mov.b64 %0, {%1, %1};" : "=l"(aa) : "f"(a));
    #pragma unroll
    for (int v = 0; v < 8; v += 2) {
        unsigned long long b, c;
        asm("mov.b64 %0, {%1, %2};" : "=l"(b) : "f"(x[v]), "f"(x[v + 1]));
        asm("mov.b64 %0, {%1, %2};" : "=l"(c) : "f"(acc[v]), "f"(acc[v + 1]));
        asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(c) : "l"(aa), "l"(b));
        asm("mov.b64 {%0, %1}, %2;" : "=f"(acc[v]), "=f"(acc[v + 1]) : "l"(c));
    }
}

// Rows of a CTA in shared memory: A[k][group][8], group g's RT rows at g ^ (k / 4)
// (a warp's stores of a thread's outputs, 4 k apart, would share a bank).
__device__ __forceinline__ int st_at(int k, int g) { return k * SUR_H + ((g ^ (k >> 2)) & 15) * 8; }

template <int RT>
__device__ __forceinline__ void st_gemm(const float* __restrict__ A, const float* __restrict__ B, int tx, int ty,
                                        float (&acc)[RT][8])
{
    #pragma unroll
    for (int r = 0; r < RT; r++)
        #pragma unroll
        for (int v = 0; v < 8; v++) acc[r][v] = 0.f;
    #pragma unroll 2
    for (int k4 = 0; k4 < SUR_H; k4 += 4) {
        const float* Ak = A + st_at(k4, ty);
        #pragma unroll
        for (int k = 0; k < 4; k++) {
            float a[8], b[8];
            *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(Ak + k * SUR_H);
            if (RT > 4) *reinterpret_cast<float4*>(a + 4) = *reinterpret_cast<const float4*>(Ak + k * SUR_H + 4);
            *reinterpret_cast<float4*>(b) = *reinterpret_cast<const float4*>(B + (k4 + k) * SUR_H + 4 * tx);
            *reinterpret_cast<float4*>(b + 4) = *reinterpret_cast<const float4*>(B + (k4 + k) * SUR_H + 64 + 4 * tx);
            #pragma unroll
            for (int r = 0; r < RT; r++) st_fma8(a[r], b, acc[r]);
        }
    }
}

// a thread's outputs to the shared rows and to out [bs][128]
template <int RT>
__device__ __forceinline__ void st_store(float* A, float* __restrict__ out, int tx, int ty, int m0, int bs,
                                         const float (&v)[RT][8], bool keep)
{
    if (keep)
        #pragma unroll
        for (int c = 0; c < 8; c++) {
            float* p = A + st_at(4 * tx + (c & 3) + 64 * (c >> 2), ty);
            #pragma unroll
            for (int r = 0; r < RT; r++) p[r] = v[r][c];
        }
    #pragma unroll
    for (int r = 0; r < RT; r++) {
        const int m = m0 + ty * RT + r;
        if (m < bs) {
            float4* o = reinterpret_cast<float4*>(out + (size_t)m * SUR_H) + tx;
            o[0] = make_float4(v[r][0], v[r][1], v[r][2], v[r][3]);
            o[16] = make_float4(v[r][4], v[r][5], v[r][6], v[r][7]);
        }
    }
}

template <int RT>
__global__ void __launch_bounds__(ST_THREADS, 1) k_sur_chain(SurTrain T)
{
    extern __shared__ __align__(16) float st_smem[];
    float* W = st_smem;                       // two 128 x 128 matrices
    float* A = st_smem + 2 * ST_HH;
    float* W4 = A + ST_HH;                    // [128][2]
    float* dy = W4 + 2 * SUR_H;               // [2][128 rows]
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4, m0 = blockIdx.x * 16 * RT, bs = T.bs;
    const size_t hs = (size_t)bs * SUR_H;
    // the layers in the order they are used: 1, 2, 3 and then 3, 2, 1 transposed
    auto load = [&](int j) {
        const float* src = j < 3 ? T.P + SUR_W1 + j * (ST_HH + SUR_H) : T.PT + (5 - j) * ST_HH;
        float* dst = W + (j & 1) * ST_HH;
        #pragma unroll 4
        for (int e = tid; e < ST_HH / 4; e += ST_THREADS) st_cp16(dst + 4 * e, src + 4 * e, true);
    };
    load(0);
    st_commit();
    load(1);
    st_commit();
    W4[tid] = T.P[SUR_W4 + tid];
    float acc[RT][8];
    {   // layer 0
        float b[8], w[3][8];
        #pragma unroll
        for (int v = 0; v < 8; v++) {
            const int c = 4 * tx + (v & 3) + 64 * (v >> 2);
            b[v] = T.P[SUR_B0 + c];
            #pragma unroll
            for (int i = 0; i < 3; i++) w[i][v] = T.P[SUR_W0 + i * SUR_H + c];
        }
        #pragma unroll
        for (int r = 0; r < RT; r++) {
            const int m = m0 + ty * RT + r;
            float x[3];
            #pragma unroll
            for (int i = 0; i < 3; i++) x[i] = m < bs ? T.x[3 * (size_t)m + i] : 0.f;
            #pragma unroll
            for (int v = 0; v < 8; v++) {
                const float s = __fmaf_rn(x[2], w[2][v], __fmaf_rn(x[1], w[1][v], __fmaf_rn(x[0], w[0][v], 0.f)));
                acc[r][v] = sur_tanh(s + b[v]);
            }
        }
        st_store<RT>(A, T.act + hs, tx, ty, m0, bs, acc, true);
    }
    #pragma unroll 1
    for (int j = 0; j < 6; j++) {
        const int l = j < 3 ? j + 1 : 6 - j;           // the layer; backward: the activations in front of it
        float4 h[RT][2];
        if (j >= 3)
            #pragma unroll
            for (int r = 0; r < RT; r++) {
                const int m = min(m0 + ty * RT + r, bs - 1);
                const float4* p = reinterpret_cast<const float4*>(T.act + l * hs + (size_t)m * SUR_H) + tx;
                h[r][0] = p[0];
                h[r][1] = p[16];
            }
        st_wait<1>();
        __syncthreads();
        st_gemm<RT>(A, W + (j & 1) * ST_HH, tx, ty, acc);
        __syncthreads();
        if (j < 4) load(j + 2);
        st_commit();
        if (j < 3) {
            #pragma unroll
            for (int v = 0; v < 8; v++) {
                const float b = T.P[SUR_B1 + j * (ST_HH + SUR_H) + 4 * tx + (v & 3) + 64 * (v >> 2)];
                #pragma unroll
                for (int r = 0; r < RT; r++) acc[r][v] = sur_tanh(acc[r][v] + b);
            }
            st_store<RT>(A, T.act + (l + 1) * hs, tx, ty, m0, bs, acc, true);
        } else {
            #pragma unroll
            for (int r = 0; r < RT; r++)
                #pragma unroll
                for (int v = 0; v < 8; v++) {
                    const float a = reinterpret_cast<const float*>(&h[r][v >> 2])[v & 3];
                    acc[r][v] = acc[r][v] * (1.f - a * a);
                }
            st_store<RT>(A, T.dz + (l - 1) * hs, tx, ty, m0, bs, acc, l > 1);
        }
        if (j != 2) continue;
        // output layer, the loss's gradient, and back through the layer
        __syncthreads();
        if (tid < 32 * RT) {
            const int o = tid & 1, row = tid >> 1, g = row / RT, r = row - g * RT, m = m0 + row;
            float s = 0.f;
            #pragma unroll 8
            for (int k = 0; k < SUR_H; k++) s = __fmaf_rn(A[st_at(k, g) + r], W4[2 * k + o], s);
            float d = 0.f;
            if (m < bs) {
                const float y = s + T.P[SUR_B4 + o];
                const float w = T.w ? T.w[m] : 1.f;
                const float e = y - T.t[2 * (size_t)m + o];
                d = 2.f * w * e / bs;
                T.act[5 * hs + 2 * (size_t)m + o] = y;
                T.dz[4 * hs + 2 * (size_t)m + o] = d;
            }
            dy[o * SUR_H + g * 8 + r] = d;
        }
        __syncthreads();
        #pragma unroll
        for (int v = 0; v < 8; v++) {
            const int c = 4 * tx + (v & 3) + 64 * (v >> 2);
            #pragma unroll
            for (int r = 0; r < RT; r++) {
                const float a = acc[r][v];
                const float s = __fmaf_rn(dy[SUR_H + ty * 8 + r], W4[2 * c + 1],
                                          __fmaf_rn(dy[ty * 8 + r], W4[2 * c], 0.f));
                acc[r][v] = s * (1.f - a * a);
            }
        }
        st_store<RT>(A, T.dz + 3 * hs, tx, ty, m0, bs, acc, true);
    }
}

// blocks [0, KS): first and last layer's weight gradients of one split;
// [KS, KS + 129): bias sums (a warp per layer and residue of 256; the output's in
// the last); then a 64 x 128 tile of one split of layer 1, 2 or 3.
__global__ void __launch_bounds__(ST_THREADS, 2) k_sur_wgrad(SurTrain T)
{
    extern __shared__ __align__(16) float st_smem[];
    const int tid = threadIdx.x, bs = T.bs, KS = T.KS;
    const size_t hs = (size_t)bs * SUR_H;
    int b = blockIdx.x;
    if (b < KS) {
        const int s0 = b * T.ksplit, s1 = min(bs, s0 + T.ksplit), c = tid & (SUR_H - 1);
        const bool first = tid < SUR_H;
        const float* v = first ? T.dz : T.act + 4 * hs;                 // [bs][128]
        const float* u = first ? T.x : T.dz + 4 * hs;                   // [bs][3] or [bs][2]
        const int nu = first ? 3 : 2;
        float a0 = 0.f, a1 = 0.f, a2 = 0.f;
        #pragma unroll 8
        for (int s = s0; s < s1; s++) {
            const float x = v[(size_t)s * SUR_H + c];
            const float* us = u + (size_t)s * nu;
            a0 = __fmaf_rn(us[0], x, a0);
            a1 = __fmaf_rn(us[1], x, a1);
            if (first) a2 = __fmaf_rn(us[2], x, a2);
        }
        if (first) {
            float* g = T.gpart + (size_t)KS * 3 * ST_HH + (size_t)b * 3 * SUR_H + c;
            g[0] = a0;
            g[SUR_H] = a1;
            g[2 * SUR_H] = a2;
        } else {
            float* g = T.gpart + (size_t)KS * (3 * ST_HH + 3 * SUR_H) + (size_t)b * 2 * SUR_H + 2 * c;
            g[0] = a0;
            g[1] = a1;
        }
        return;
    }
    b -= KS;
    if (b < 128) {
        const int warp = b * 8 + (tid >> 5), l = warp >> 8, t = warp & 255;
        const float4* d = reinterpret_cast<const float4*>(T.dz + l * hs) + (tid & 31);
        float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
        #pragma unroll 8
        for (int r = t; r < bs; r += 256) {
            const float4 v = d[(size_t)r * (SUR_H / 4)];
            s.x += v.x; s.y += v.y; s.z += v.z; s.w += v.w;
        }
        reinterpret_cast<float4*>(T.cpart + warp * SUR_H)[tid & 31] = s;
        return;
    }
    if (b == 128) {
        const float2* d = reinterpret_cast<const float2*>(T.dz + 4 * hs);
        float2 s = make_float2(0.f, 0.f);
        #pragma unroll 8
        for (int r = tid; r < bs; r += 256) { const float2 v = d[r]; s.x += v.x; s.y += v.y; }
        reinterpret_cast<float2*>(T.cpart + 4 * 256 * SUR_H)[tid] = s;
        return;
    }
    b -= 129;
    const int half = b & 1, z = (b >> 1) % KS, l = (b >> 1) / KS + 1;
    const int tx = tid & 15, ty = tid >> 4;
    const int s0 = z * T.ksplit, s1 = min(bs, s0 + T.ksplit), nk = (s1 - s0 + ST_WG_K - 1) / ST_WG_K;
    const float* av = T.act + l * hs + 64 * half;
    const float* dv = T.dz + l * hs;
    auto load = [&](int q) {
        float* st = st_smem + (q % 3) * ST_WG_STAGE;
        #pragma unroll
        for (int e = tid; e < ST_WG_K * 48; e += ST_THREADS) {
            const int k = e / 48, w = e - k * 48, s = s0 + q * ST_WG_K + k;
            const bool ok = s < s1;
            const size_t row = (size_t)(ok ? s : s0) * SUR_H;
            if (w < 16) st_cp16(st + k * 64 + 4 * w, av + row + 4 * w, ok);
            else st_cp16(st + ST_WG_K * 64 + k * SUR_H + 4 * (w - 16), dv + row + 4 * (w - 16), ok);
        }
    };
    float acc[4][8] = {};
    if (nk > 0) load(0);
    st_commit();
    if (nk > 1) load(1);
    st_commit();
    for (int q = 0; q < nk; q++) {
        st_wait<1>();
        __syncthreads();
        if (q + 2 < nk) load(q + 2);
        st_commit();
        const float* Aq = st_smem + (q % 3) * ST_WG_STAGE;
        const float* Bq = Aq + ST_WG_K * 64;
        #pragma unroll 8
        for (int k = 0; k < ST_WG_K; k++) {
            float a[4], v[8];
            *reinterpret_cast<float4*>(a) = *reinterpret_cast<const float4*>(Aq + k * 64 + 4 * ty);
            *reinterpret_cast<float4*>(v) = *reinterpret_cast<const float4*>(Bq + k * SUR_H + 4 * tx);
            *reinterpret_cast<float4*>(v + 4) = *reinterpret_cast<const float4*>(Bq + k * SUR_H + 64 + 4 * tx);
            #pragma unroll
            for (int r = 0; r < 4; r++) st_fma8(a[r], v, acc[r]);
        }
    }
    float* g = T.gpart + ((size_t)(l - 1) * KS + z) * ST_HH + (64 * half + 4 * ty) * SUR_H + 4 * tx;
    #pragma unroll
    for (int r = 0; r < 4; r++) {
        *reinterpret_cast<float4*>(g + r * SUR_H) = make_float4(acc[r][0], acc[r][1], acc[r][2], acc[r][3]);
        *reinterpret_cast<float4*>(g + r * SUR_H + 64) = make_float4(acc[r][4], acc[r][5], acc[r][6], acc[r][7]);
    }
}

// Layer of parameter i and its place in it (weights, then biases).
__device__ __forceinline__ void st_place(int i, int& l, int& e)
{
    if (i < SUR_W1) { l = 0; e = i; }
    else if (i < SUR_W4) { l = 1 + (i - SUR_W1) / (ST_HH + SUR_H); e = (i - SUR_W1) % (ST_HH + SUR_H); }
    else { l = 4; e = i - SUR_W4; }
}

__device__ __forceinline__ void st_adam(const SurTrain& T, int i, float gi, bool adam, float lr, float b1, float b2,
                                        float c1, float c2)
{
    T.grad[i] = gi;
    if (!adam) return;
    const float a = b1 * T.m1[i] + (1.f - b1) * gi;
    const float b = b2 * T.m2[i] + (1.f - b2) * gi * gi;
    T.m1[i] = a;
    T.m2[i] = b;
    const float p = T.P[i] - lr * (a * c1) / (sqrtf(b * c2) + 1e-8f);
    T.P[i] = p;
    int l, e;
    st_place(i, l, e);
    if (l >= 1 && l <= 3 && e < ST_HH) T.PT[(l - 1) * ST_HH + (e & (SUR_H - 1)) * SUR_H + e / SUR_H] = p;
}

// blocks [0, ceil(SUR_NP / 256)): a thread per weight; then a warp per bias
#define ST_UPDATE_BLOCKS ((SUR_NP + 255) / 256)
__global__ void __launch_bounds__(ST_THREADS) k_sur_update(SurTrain T, int adam, float lr, float b1, float b2, float c1,
                                                           float c2)
{
    if (blockIdx.x < ST_UPDATE_BLOCKS) {
        const int i = blockIdx.x * ST_THREADS + threadIdx.x;
        if (i >= SUR_NP) return;
        int l, e;
        st_place(i, l, e);
        const int nw = l == 0 ? 3 * SUR_H : l == 4 ? 2 * SUR_H : ST_HH;
        if (e >= nw) return;                                     // a bias
        const float* g = T.gpart + (l == 0 ? (size_t)T.KS * 3 * ST_HH
                                           : l == 4 ? (size_t)T.KS * (3 * ST_HH + 3 * SUR_H)
                                                    : (size_t)(l - 1) * T.KS * ST_HH) + e;
        float s = 0.f;
        #pragma unroll 8
        for (int z = 0; z < T.KS; z++) s += g[(size_t)z * nw];
        st_adam(T, i, s, adam, lr, b1, b2, c1, c2);
        return;
    }
    const int bias = (blockIdx.x - ST_UPDATE_BLOCKS) * 8 + (threadIdx.x >> 5), lane = threadIdx.x & 31;
    if (bias >= 4 * SUR_H + 2) return;
    const int l = bias / SUR_H, c = bias - l * SUR_H, no = l == 4 ? 2 : SUR_H;
    const float* p = T.cpart + l * 256 * SUR_H + c;
    float r[8];
    #pragma unroll
    for (int j = 0; j < 8; j++) r[j] = p[(lane + 32 * j) * no];
    // the tree over the 256 residues: 128 and 64 and 32 apart in the lane, then across
    #pragma unroll
    for (int o = 4; o > 0; o >>= 1)
        #pragma unroll
        for (int j = 0; j < o; j++) r[j] += r[j + o];
    #pragma unroll
    for (int o = 16; o > 0; o >>= 1) r[0] += __shfl_down_sync(0xffffffffu, r[0], o);
    if (lane == 0)
        st_adam(T, (l == 0 ? SUR_B0 : l == 4 ? SUR_B4 : SUR_B1 + (l - 1) * (ST_HH + SUR_H)) + c, r[0], adam, lr, b1, b2,
                c1, c2);
}

__global__ void k_sur_transpose(const float* __restrict__ P, float* __restrict__ PT)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= 3 * ST_HH) return;
    const int l = i / ST_HH, e = i - l * ST_HH;
    PT[l * ST_HH + (e & (SUR_H - 1)) * SUR_H + e / SUR_H] = P[SUR_W1 + l * (ST_HH + SUR_H) + e];
}

template <int RT>
static cudaError_t st_chain(const SurTrain& T, cudaStream_t s)
{
    cudaError_t e = cudaFuncSetAttribute(k_sur_chain<RT>, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_CHAIN_SMEM);
    if (e == cudaSuccess) k_sur_chain<RT><<<(T.bs + 16 * RT - 1) / (16 * RT), ST_THREADS, ST_CHAIN_SMEM, s>>>(T);
    return e;
}

// Forward and backward pass: the gradients' parts, and with lpart the loss's.
// RT: a CTA's time goes with RT + 1 (the weights' copies, the output layer), so
// the one of 2 to 8 with the fewest waves x (RT + 1) -- 7 for 16,384 rows: 147 CTAs on
// 152 SMs, 130 us a step (8, as many waves, 136; 4, two waves, 147).  With 2, 4, 7 and 8
// alone 10,240 rows took 111 us (5 rows: 92), 12,288 120 (6: 110), 24,000 275 (5: 192).
static cudaError_t st_fwd_bwd(const SurTrain& T, int sms, int mse_blocks, cudaStream_t s)
{
    static cudaError_t (*const chain[7])(const SurTrain&, cudaStream_t) = {st_chain<2>, st_chain<3>, st_chain<4>, st_chain<5>,
                                                                           st_chain<6>, st_chain<7>, st_chain<8>};
    int rt = 8;
    long best = 1L << 60;
    for (int r = 2; r <= 8; r++) {
        const long tiles = (T.bs + 16 * r - 1) / (16 * r), cost = (tiles + sms - 1) / sms * (r + 1);
        if (cost < best) { best = cost; rt = r; }
    }
    cudaError_t e = chain[rt - 2](T, s);
    if (e != cudaSuccess) return e;
    if (T.lpart)
        k_sur_mse<<<mse_blocks, 256, 0, s>>>(T.bs, T.act + 5 * (size_t)T.bs * SUR_H, T.t, T.w,
                                             T.dz + 4 * (size_t)T.bs * SUR_H, T.lpart);
    e = cudaFuncSetAttribute(k_sur_wgrad, cudaFuncAttributeMaxDynamicSharedMemorySize, ST_WG_SMEM);
    if (e != cudaSuccess) return e;
    k_sur_wgrad<<<T.KS + 129 + 6 * T.KS, ST_THREADS, ST_WG_SMEM, s>>>(T);
    return cudaSuccess;
}

static void st_update(const SurTrain& T, bool adam, float lr, float b1, float b2, float c1, float c2, cudaStream_t s)
{
    k_sur_update<<<ST_UPDATE_BLOCKS + (4 * SUR_H + 2 + 7) / 8, ST_THREADS, 0, s>>>(T, adam ? 1 : 0, lr, b1, b2, c1, c2);
}

}  // namespace qlpix
