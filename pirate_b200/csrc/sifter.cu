// sifter.cu -- candidate patches and the sifter MLP (see sifter.hpp).

#include "sifter.hpp"

#include <cuda_bf16.h>
#include <cuda_fp16.h>

#include <cmath>
#include <cstring>
#include <random>
#include <stdexcept>
#include <string>

namespace pb2 {

#define SF_CHECK(x) do { cudaError_t _e = (x); if (_e != cudaSuccess) \
    throw std::runtime_error(std::string("sifter: " #x ": ") + cudaGetErrorString(_e)); } while (0)

static void sf_check_launch(const char *what)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess) throw std::runtime_error(std::string(what) + ": launch failed: " + cudaGetErrorString(e));
}

template<typename T> __device__ __forceinline__ float sf_to_f(T x);
template<> __device__ __forceinline__ float sf_to_f<float>(float x) { return x; }
template<> __device__ __forceinline__ float sf_to_f<__half>(__half x) { return __half2float(x); }
template<> __device__ __forceinline__ float sf_to_f<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

// ---------------------------------------------------------------------------------------------
// Patches. One block per batch beam; thread (w, j) = (threadIdx.x / 32, threadIdx.x % 32) computes the
// width-2^w trailing boxcar ending at window time j for the 9 fine DMs.

template<typename Ts>
__global__ void __launch_bounds__(kPatchW * 32) patch_kernel(PatchArgs a)
{
    const int b = blockIdx.x;
    const int w = threadIdx.x >> 5, j = threadIdx.x & 31;
    __half *out = (__half *) a.patches + (long) b * kPatchLen;
    const float pk = a.peak[b];
    const int it = a.tree[b];
    const bool ok = (pk >= a.threshold) && (it >= 0) && (it < a.ntrees);
    if (threadIdx.x == 0) a.valid[b] = ok ? 1 : 0;
    if (!ok) {
        for (int d = 0; d < kPatchDm; d++) out[(d * kPatchT + j) * kPatchW + w] = __float2half_rn(0.0f);
        return;
    }
    const PatchTree &t = a.t[it];
    const uint32_t tok = a.token[b];
    const int m = (tok >> 16) & 0xffff, p = (tok >> 8) & 0xff, tf = tok & 0xff;
    const int l = p ? (p - 1) / 3 : 0;
    const int dt = min(t.Dcore, 1 << l);
    const long s0 = (a.chunk_ctr ? *a.chunk_ctr : a.ichunk) * t.nt_ds;
    // Last sample of the winning trial (the decode_argmax convention), placed at window time 23,
    // shifted so that the window ends inside the chunk.
    const long tend = s0 + (long) a.itime[b] * t.Dout + tf + dt - 1;
    long last = tend + (kPatchT - 1 - kPatchPeakAt);
    if (last > s0 + t.nt_ds - 1) last = s0 + t.nt_ds - 1;
    const long sj = last - (kPatchT - 1) + j;
    const int R = t.pf_rank;
    // Fine DM of the winning multiplet: coarse dm * 2^pf_rank + its fine offset (full band).
    int d0 = 0;
    for (int dd = 0; dd < (1 << R); dd++)
        if (t.d_to_m[dd] == m) d0 = dd;
    const long f0 = (long) a.idm[b] * (1 << R) + d0;
    const long nfine = (long) t.ndm_out << R;
    const long mask = t.pf_cap - 1;
    const int width = 1 << w;
    const float norm = rsqrtf((float) width);
    const int itw = a.itime[b] / (t.nt_out / t.nt_wt);
    const int dwds = t.ndm_out / t.ndm_wt;
    for (int d = 0; d < kPatchDm; d++) {
        const long f = f0 - kPatchDm / 2 + d;
        float v = 0.0f;
        if (f >= 0 && f < nfine) {
            const int mm = t.d_to_m[f & ((1 << R) - 1)];
            if (mm >= 0) {
                const Ts *row = (const Ts *) t.pf + (((long) (a.beam0 + b) * t.ndm_out + (f >> R)) * t.M + mm) * t.pf_cap;
                const float scale = t.wt[(((long) b * t.ndm_wt + (f >> R) / dwds) * t.nt_wt + itw) * t.P * t.N + t.nfull];
                float s = 0.0f;
                for (int k = 0; k < width; k++) s += sf_to_f(row[(sj - k) & mask]);
                v = 8.0f * asinhf(s * scale * norm * 0.125f);
            }
        }
        out[(d * kPatchT + j) * kPatchW + w] = __float2half_rn(v);
    }
}

void launch_patches(const PatchArgs &a, int dtype, cudaStream_t s)
{
    if (a.B <= 0) return;
    if (a.ntrees <= 0 || a.ntrees > kPatchMaxTrees) throw std::runtime_error("patches: bad number of trees");
    if (dtype == 0) patch_kernel<float><<<a.B, kPatchW * 32, 0, s>>>(a);
    else if (dtype == 1) patch_kernel<__half><<<a.B, kPatchW * 32, 0, s>>>(a);
    else if (dtype == 2) patch_kernel<__nv_bfloat16><<<a.B, kPatchW * 32, 0, s>>>(a);
    else throw std::runtime_error("patches: bad dtype");
    sf_check_launch("patch_kernel");
}

__global__ void mask_scores_kernel(const float *logits, const int *valid, float *scores, int n)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) scores[i] = valid[i] ? logits[i] : -INFINITY;
}

void launch_mask_scores(const float *logits, const int *valid, float *scores, int n, cudaStream_t s)
{
    if (n <= 0) return;
    mask_scores_kernel<<<(n + 127) / 128, 128, 0, s>>>(logits, valid, scores, n);
    sf_check_launch("mask_scores_kernel");
}

// ---------------------------------------------------------------------------------------------
// The MLP on the tensor cores: bf16 operands, FP32 accumulation (mma.sync m16n8k16). At 1 MFLOP per candidate and
// at most 1024 candidates the work is bound by latency, so the kernels are few and wide. (One GEMM kernel per product,
// its K loop of 32-wide steps unpipelined, took about 24 launches and 620 us per training step of 512, and 0.4 ms for
// the 8 candidates of a chunk; these take 3 launches and about 120 us with the host's part, and 38 us with the patches.)
//   layer1_kernel  Z1 = X W1^T + b1, H1 = bf16(relu(Z1)): 32 x 32 tiles, K in chunks of 64 through a cp.async
//                  pipeline
//   head_kernel    16 candidates per block: layers 2 and 3, and in training everything between the logits and
//                  the weight gradients (loss terms, g, g2, g1)
//   wgrad_kernel   dW1 = g1^T X, dW2 = g2^T H1 and dW3 = g^T H2 in 64 x 64 tiles, the bias gradients and the loss,
//                  with the Adam step in the epilogue
// Every product is one chain of k16 steps from K = 0 and every bias gradient one chain over the candidates, whatever
// the batch size: a hidden value near a rounding boundary of bf16 rounds another way after another order of its sum, so
// a candidate's score would depend on the batch that it is scored in, and a training run on the split chosen.

constexpr int kIn = kMlpIn, kH1 = kMlpH1, kH2 = kMlpH2;
constexpr int kKc = 64, kKPitch = kKc + 8;    // K chunk; padded row of a staged tile (ldmatrix without bank conflicts)
constexpr int kStages = 3;                    // wgrad_kernel
constexpr int kL1Stages = 5;                  // layer1_kernel: its 27 chunks are a serial chain; 46 KB of shared memory
constexpr int kHeadRows = 16;

__device__ __forceinline__ void mma_bf16(float (&c)[4], const uint32_t (&a)[4], uint32_t b0, uint32_t b1)
{
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0,%1,%2,%3}, {%4,%5,%6,%7}, {%8,%9}, {%0,%1,%2,%3};\n"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a[0]), "r"(a[1]), "r"(a[2]), "r"(a[3]), "r"(b0), "r"(b1));
}
__device__ __forceinline__ void ldsm4(uint32_t (&r)[4], const void *p)
{
    const unsigned a = (unsigned) __cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
__device__ __forceinline__ void ldsm4t(uint32_t (&r)[4], const void *p)
{
    const unsigned a = (unsigned) __cvta_generic_to_shared(p);
    asm volatile("ldmatrix.sync.aligned.m8n8.x4.trans.shared.b16 {%0,%1,%2,%3}, [%4];\n" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(a) : "memory");
}
// 16-byte asynchronous copy, zeros when !ok (the source is then not read).
__device__ __forceinline__ void cp16(void *dst, const void *src, bool ok)
{
    const unsigned d = (unsigned) __cvta_generic_to_shared(dst);
    const int n = ok ? 16 : 0;
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16, %2;\n" :: "r"(d), "l"(src), "r"(n) : "memory");
}
// Eight 16-bit values of an input row that need not start on a 16-byte boundary.
__device__ __forceinline__ void copy8(uint16_t *dst, const uint16_t *src, bool ok, bool aligned)
{
    if (aligned) {
        cp16(dst, src, ok);
    } else {
#pragma unroll
        for (int i = 0; i < 8; i++) dst[i] = ok ? src[i] : 0;
    }
}
__device__ __forceinline__ uint32_t half2_to_bf162(uint32_t h)
{
    const float2 f = __half22float2(*(const __half2 *) &h);
    const __nv_bfloat162 b = __floats2bfloat162_rn(f.x, f.y);
    return *(const uint32_t *) &b;
}
__device__ __forceinline__ float relu(float x) { return (x < 0.0f) ? 0.0f : x; }   // NaN passes
__device__ __forceinline__ float bf_round(float x) { return __bfloat162float(__float2bfloat16_rn(x)); }
__device__ __forceinline__ uint16_t bf_bits(float x)
{
    const __nv_bfloat16 h = __float2bfloat16_rn(x);
    return *(const uint16_t *) &h;
}
__device__ __forceinline__ float bf_float(uint16_t b) { return __uint_as_float(uint32_t(b) << 16); }

template<int N> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" :: "n"(N) : "memory"); }
__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }

struct Layer1Args
{
    const uint16_t *x, *w;   // fp16 (n, kIn), bf16 (kH1, kIn)
    const float *bias;
    int n, aligned;
    float *z;
    uint16_t *h;
};

// Grid (kH1 / 32, row blocks). The sum over K is not split over blocks (see above).
__global__ void __launch_bounds__(128) layer1_kernel(Layer1Args g)
{
    __shared__ __align__(16) uint16_t As[kL1Stages][32][kKPitch], Bs[kL1Stages][32][kKPitch];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int n0 = blockIdx.x * 32, m0 = blockIdx.y * 32;
    constexpr int NC = kIn / kKc;
    auto load = [&](int c) {
        if (c < NC) {
            const int st = c % kL1Stages;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int i = tid + 128 * j, r = i >> 3, k = (i & 7) * 8;
                const bool ok = m0 + r < g.n;
                copy8(&As[st][r][k], g.x + (long) (ok ? m0 + r : 0) * kIn + c * kKc + k, ok, g.aligned);
                cp16(&Bs[st][r][k], g.w + (long) (n0 + r) * kIn + c * kKc + k, true);
            }
        }
        cp_commit();
    };
    for (int c = 0; c < kL1Stages - 1; c++) load(c);
    const int wm = (warp >> 1) * 16, wn = (warp & 1) * 16;
    float acc[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
    for (int c = 0; c < NC; c++) {
        cp_wait<kL1Stages - 2>();
        __syncthreads();
        load(c + kL1Stages - 1);   // into the buffer that was read before this barrier
        const int st = c % kL1Stages;
#pragma unroll
        for (int ks = 0; ks < kKc; ks += 16) {
            uint32_t a[4], b[4];
            ldsm4(a, &As[st][wm + (lane & 15)][ks + (lane >> 4) * 8]);
            ldsm4(b, &Bs[st][wn + (lane >> 4) * 8 + (lane & 7)][ks + ((lane >> 3) & 1) * 8]);
#pragma unroll
            for (int i = 0; i < 4; i++) a[i] = half2_to_bf162(a[i]);
            mma_bf16(acc[0], a, b[0], b[1]);
            mma_bf16(acc[1], a, b[2], b[3]);
        }
    }
#pragma unroll
    for (int t = 0; t < 2; t++)
#pragma unroll
        for (int h = 0; h < 2; h++) {
            const int r = m0 + wm + (lane >> 2) + 8 * h, c = n0 + wn + t * 8 + (lane & 3) * 2;
            if (r >= g.n) continue;
            const float v0 = acc[t][2 * h] + g.bias[c], v1 = acc[t][2 * h + 1] + g.bias[c + 1];
            *(float2 *) (g.z + (long) r * kH1 + c) = make_float2(v0, v1);
            *(uint32_t *) (g.h + (long) r * kH1 + c) = uint32_t(bf_bits(relu(v0))) | (uint32_t(bf_bits(relu(v1))) << 16);
        }
}

constexpr int kGPitch = 8;   // bf16 per row of the operand gb: g, then zeros (one 16-byte copy)

struct HeadArgs
{
    const uint16_t *h1, *w2, *w3;   // bf16
    const float *z1, *b2, *b3;
    int n;
    float *logits;           // inference
    const float *labels;     // training (null: inference)
    // Training: gradients of the logits, Z2 and Z1 in fp32 (n), (n, kH2), (n, kH1) for the bias gradients, and rounded
    // to bf16 as the products take them; H2 as an operand; each candidate's loss term.
    float *g, *g2, *g1, *ls;
    uint16_t *gb, *g2b, *g1b, *h2;
};

struct HeadSmem
{
    uint16_t h1[kHeadRows][kH1 + 8];
    uint16_t w2[kH2][kH1 + 8];
    float z2[kHeadRows][kH2 + 4];
    uint16_t h2[kHeadRows][kH2 + 8];
    uint16_t g2[kHeadRows][kH2 + 8];
    uint16_t w3[kH2];
    float g[kHeadRows];
};

__global__ void __launch_bounds__(256) head_kernel(HeadArgs g)
{
    extern __shared__ __align__(16) unsigned char head_sm[];
    HeadSmem &s = *(HeadSmem *) head_sm;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    const int r0 = blockIdx.x * kHeadRows;
    for (int i = tid; i < kHeadRows * (kH1 / 8); i += 256) {
        const int r = i / (kH1 / 8), k = i % (kH1 / 8) * 8;
        const bool ok = r0 + r < g.n;
        cp16(&s.h1[r][k], g.h1 + (long) (ok ? r0 + r : 0) * kH1 + k, ok);
    }
    for (int i = tid; i < kH2 * (kH1 / 8); i += 256) {
        const int r = i / (kH1 / 8), k = i % (kH1 / 8) * 8;
        cp16(&s.w2[r][k], g.w2 + (long) r * kH1 + k, true);
    }
    cp_commit();
    if (tid < kH2) s.w3[tid] = g.w3[tid];
    cp_wait<0>();
    __syncthreads();
    {
        // Z2 = H1 W2^T + b2: warp w takes 16 columns
        float acc[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
        const int c0 = warp * 16;
#pragma unroll
        for (int ks = 0; ks < kH1; ks += 16) {
            uint32_t a[4], b[4];
            ldsm4(a, &s.h1[lane & 15][ks + (lane >> 4) * 8]);
            ldsm4(b, &s.w2[c0 + (lane >> 4) * 8 + (lane & 7)][ks + ((lane >> 3) & 1) * 8]);
            mma_bf16(acc[0], a, b[0], b[1]);
            mma_bf16(acc[1], a, b[2], b[3]);
        }
#pragma unroll
        for (int t = 0; t < 2; t++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int c = c0 + t * 8 + (lane & 3) * 2 + (q & 1);
                const int r = (lane >> 2) + (q >> 1) * 8;
                const float z = acc[t][q] + g.b2[c];
                s.z2[r][c] = z;
                s.h2[r][c] = bf_bits(relu(z));
            }
    }
    __syncthreads();
    if (warp == 0) {
        // logit = H2 W3^T + b3: one tile, W3 its first column
        float acc[4] = {0, 0, 0, 0};
#pragma unroll
        for (int ks = 0; ks < kH2; ks += 16) {
            uint32_t a[4], b[2] = {0, 0};
            ldsm4(a, &s.h2[lane & 15][ks + (lane >> 4) * 8]);
            if (lane < 4) {
                b[0] = *(const uint32_t *) &s.w3[ks + lane * 2];
                b[1] = *(const uint32_t *) &s.w3[ks + 8 + lane * 2];
            }
            mma_bf16(acc, a, b[0], b[1]);
        }
        if ((lane & 3) == 0) {
#pragma unroll
            for (int h = 0; h < 2; h++) {
                const int row = (lane >> 2) + 8 * h, r = r0 + row;
                const bool live = r < g.n;
                const float logit = acc[2 * h] + g.b3[0];
                if (!g.labels) {
                    if (live) g.logits[r] = logit;
                    continue;
                }
                // Mean binary cross-entropy; g = (sigmoid(z) - y) / n
                float gi = 0.0f;
                if (live) {
                    const float y = g.labels[r];
                    const float sig = 1.0f / (1.0f + expf(-logit));
                    gi = (sig - y) / (float) g.n;
                    g.g[r] = gi;
                    *(uint4 *) (g.gb + (long) r * kGPitch) = make_uint4(bf_bits(gi), 0, 0, 0);
                    g.ls[r] = fmaxf(logit, 0.0f) - logit * y + log1pf(expf(-fabsf(logit)));
                }
                s.g[row] = bf_round(gi);
            }
        }
    }
    if (!g.labels) return;
    __syncthreads();
    for (int i = tid; i < kHeadRows * kH2; i += 256) {
        // g2 = (g W3) masked by Z2 > 0 (a product of two bf16 values is exact in fp32)
        const int row = i / kH2, c = i % kH2;
        const float g2 = (s.z2[row][c] > 0.0f) ? s.g[row] * bf_float(s.w3[c]) : 0.0f;
        const uint16_t h = bf_bits(g2);
        s.g2[row][c] = h;
        if (r0 + row < g.n) {
            const long o = (long) (r0 + row) * kH2 + c;
            g.g2[o] = g2;
            g.g2b[o] = h;
            g.h2[o] = s.h2[row][c];
        }
    }
    __syncthreads();
    // g1 = (g2 W2) masked by Z1 > 0: warp w takes 32 columns
    float acc[4][4];
#pragma unroll
    for (int t = 0; t < 4; t++)
#pragma unroll
        for (int q = 0; q < 4; q++) acc[t][q] = 0.0f;
    const int c0 = warp * 32;
#pragma unroll
    for (int ks = 0; ks < kH2; ks += 16) {
        uint32_t a[4], b[4];
        ldsm4(a, &s.g2[lane & 15][ks + (lane >> 4) * 8]);
#pragma unroll
        for (int p = 0; p < 2; p++) {
            ldsm4t(b, &s.w2[ks + (lane & 15)][c0 + p * 16 + (lane >> 4) * 8]);
            mma_bf16(acc[2 * p], a, b[0], b[1]);
            mma_bf16(acc[2 * p + 1], a, b[2], b[3]);
        }
    }
#pragma unroll
    for (int t = 0; t < 4; t++) {
        const int c = c0 + t * 8 + (lane & 3) * 2;
#pragma unroll
        for (int hh = 0; hh < 2; hh++) {
            const int r = r0 + (lane >> 2) + hh * 8;
            if (r < g.n) {
                const long o = (long) r * kH1 + c;
                const float2 z = *(const float2 *) (g.z1 + o);
                const float v0 = (z.x > 0.0f) ? acc[t][2 * hh] : 0.0f, v1 = (z.y > 0.0f) ? acc[t][2 * hh + 1] : 0.0f;
                *(float2 *) (g.g1 + o) = make_float2(v0, v1);
                *(uint32_t *) (g.g1b + o) = uint32_t(bf_bits(v0)) | (uint32_t(bf_bits(v1)) << 16);
            }
        }
    }
}

struct WgradArgs
{
    const uint16_t *g1b, *g2b, *gb, *h1, *h2, *x;   // bf16 (n, kH1), (n, kH2), (n, kGPitch), (n, kH1), (n, kH2); fp16 (n, kIn)
    const float *g1, *g2, *g, *ls;
    int n, aligned;
    float *loss;
    float *grad;                        // null: Adam step instead
    float *w, *m, *v;                   // fp32 parameters and moments
    uint16_t *wb;                       // bf16 copies of W1, W2, W3
    float lr, c1, c2;
};

static constexpr long kW1n = long(kMlpH1) * kMlpIn, kW2n = long(kMlpH2) * kMlpH1;
static constexpr long oW1 = 0, oB1 = oW1 + kW1n, oW2 = oB1 + kMlpH1, oB2 = oW2 + kW2n, oW3 = oB2 + kMlpH2, oB3 = oW3 + kMlpH2;
static constexpr long kNparams = oB3 + 1;
static constexpr long bW1 = 0, bW2 = kW1n, bW3 = kW1n + kW2n, kNbf16 = kW1n + kW2n + kMlpH2;

// The gradient gi of parameter i (bf16 copy at wb[ib], ib < 0: none): stored, or one Adam step (0.9, 0.999, 1e-8).
__device__ __forceinline__ void take_grad(const WgradArgs &g, long i, long ib, float gi)
{
    if (g.grad) {
        g.grad[i] = gi;
        return;
    }
    const float mi = 0.9f * g.m[i] + 0.1f * gi;
    const float vi = 0.999f * g.v[i] + 0.001f * gi * gi;
    g.m[i] = mi;
    g.v[i] = vi;
    const float wi = g.w[i] - g.lr * (mi / g.c1) / (sqrtf(vi / g.c2) + 1.0e-8f);
    g.w[i] = wi;
    if (ib >= 0) g.wb[ib] = bf_bits(wi);
}

constexpr int kWgK = 32;                             // candidates per pipeline step
constexpr int kWgTiles1 = (kMlpH1 / 64) * (kMlpIn / 64), kWgTiles2 = (kMlpH2 / 64) * (kMlpH1 / 64), kWgTiles3 = kMlpH2 / 64;
constexpr int kWgTiles = kWgTiles1 + kWgTiles2 + kWgTiles3;
constexpr int kWgBias = kMlpH1 / 128 + kMlpH2 / 128 + 1;   // blocks of 128 bias gradients, and one for db3 and the loss
static_assert(kMlpH1 % 128 == 0 && kMlpH2 % 128 == 0, "bias blocks");

// Sum over the candidates of x[i * pitch], in order; the next 32 are loaded while 32 are added.
__device__ __forceinline__ float chain_sum(const float *x, long pitch, int n)
{
    float v = 0.0f, a[32], b[32];
    auto load = [&](float (&o)[32], int i0) {
#pragma unroll
        for (int i = 0; i < 32; i++) o[i] = (i0 + i < n) ? x[(long) (i0 + i) * pitch] : 0.0f;
    };
    load(a, 0);
    for (int i0 = 0; i0 < n; i0 += 32) {
        load(b, i0 + 32);
#pragma unroll
        for (int i = 0; i < 32; i++) {
            v += a[i];
            a[i] = b[i];
        }
    }
    return v;
}

// Bias gradients and the loss (block 'blk' of kWgBias).
__device__ __forceinline__ void wgrad_bias(const WgradArgs &g, int blk, int tid)
{
    constexpr int N1 = kMlpH1 / 128, N2 = kMlpH2 / 128;
    if (blk < N1) {
        take_grad(g, oB1 + blk * 128 + tid, -1, chain_sum(g.g1 + blk * 128 + tid, kH1, g.n));
        return;
    }
    if (blk < N1 + N2) {
        blk -= N1;
        take_grad(g, oB2 + blk * 128 + tid, -1, chain_sum(g.g2 + blk * 128 + tid, kH2, g.n));
        return;
    }
    // db3 by the last warp; the loss as a sum per 32 candidates, then over those (at most 1024 candidates).
    __shared__ float red[32];
    const int lane = tid & 31, warp = tid >> 5;
    for (int q = warp; q < 32; q += 4) {
        float v = (q * 32 + lane < g.n) ? g.ls[q * 32 + lane] : 0.0f;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) red[q] = v;
    }
    __syncthreads();
    if (warp == 0) {
        float v = red[lane];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) g.loss[0] = v / (float) g.n;
    } else if (tid == 96) {
        take_grad(g, oB3, -1, chain_sum(g.g, 1, g.n));
    }
}

// C(m, c) = sum_k A[k][m] B[k][c] over the n candidates, 64 x 64 tiles, four warps of 32 x 32; operands are read
// as they lie (candidates in rows) and transposed by ldmatrix. dW3 is row 0 of its tiles.
__global__ void __launch_bounds__(128) wgrad_kernel(WgradArgs g)
{
    __shared__ __align__(16) uint16_t As[kStages][kWgK][kKPitch], Bs[kStages][kWgK][kKPitch];
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5;
    int blk = blockIdx.x;
    if (blk >= kWgTiles) {
        wgrad_bias(g, blk - kWgTiles, tid);
        return;
    }
    const bool first = blk < kWgTiles1, third = blk >= kWgTiles1 + kWgTiles2;
    blk -= first ? 0 : third ? kWgTiles1 + kWgTiles2 : kWgTiles1;
    const int lda = first ? kH1 : third ? kGPitch : kH2, ldb = first ? kIn : third ? kH2 : kH1;
    const int tn = ldb / 64, m0 = blk / tn * 64, c0 = blk % tn * 64;
    const int na = third ? kGPitch : 64;   // columns of A in memory; zeros beyond
    const uint16_t *A = first ? g.g1b : third ? g.gb : g.g2b, *B = first ? g.x : third ? g.h2 : g.h1;
    const bool al = first ? g.aligned : true;
    const int nk = (g.n + kWgK - 1) / kWgK;
    auto load = [&](int c) {
        if (c < nk) {
            const int st = c % kStages;
#pragma unroll
            for (int j = 0; j < 2; j++) {
                const int i = tid + 128 * j, r = i >> 3, k = (i & 7) * 8;
                const bool ok = c * kWgK + r < g.n;
                const long rr = ok ? c * kWgK + r : 0;
                cp16(&As[st][r][k], A + rr * lda + (k < na ? m0 + k : 0), ok && k < na);
                copy8(&Bs[st][r][k], B + rr * ldb + c0 + k, ok, al);
            }
        }
        cp_commit();
    };
    for (int c = 0; c < kStages - 1; c++) load(c);
    const int wm = (warp >> 1) * 32, wn = (warp & 1) * 32;
    float acc[2][4][4];
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int t = 0; t < 4; t++)
#pragma unroll
            for (int q = 0; q < 4; q++) acc[i][t][q] = 0.0f;
    for (int c = 0; c < nk; c++) {
        cp_wait<kStages - 2>();
        __syncthreads();
        load(c + kStages - 1);
        const int st = c % kStages;
#pragma unroll
        for (int ks = 0; ks < kWgK; ks += 16) {
            uint32_t a[2][4], b[2][4];
#pragma unroll
            for (int i = 0; i < 2; i++) {
                ldsm4t(a[i], &As[st][ks + (lane >> 4) * 8 + (lane & 7)][wm + i * 16 + ((lane >> 3) & 1) * 8]);
                ldsm4t(b[i], &Bs[st][ks + (lane & 15)][wn + i * 16 + (lane >> 4) * 8]);
                if (first) {
#pragma unroll
                    for (int q = 0; q < 4; q++) b[i][q] = half2_to_bf162(b[i][q]);
                }
            }
#pragma unroll
            for (int i = 0; i < 2; i++)
#pragma unroll
                for (int p = 0; p < 2; p++) {
                    mma_bf16(acc[i][2 * p], a[i], b[p][0], b[p][1]);
                    mma_bf16(acc[i][2 * p + 1], a[i], b[p][2], b[p][3]);
                }
        }
    }
    const long o = first ? oW1 : third ? oW3 : oW2, ob = first ? bW1 : third ? bW3 : bW2;
#pragma unroll
    for (int i = 0; i < 2; i++)
#pragma unroll
        for (int t = 0; t < 4; t++)
#pragma unroll
            for (int q = 0; q < 4; q++) {
                const int m = m0 + wm + i * 16 + (lane >> 2) + (q >> 1) * 8;
                const long e = (long) m * ldb + c0 + wn + t * 8 + (lane & 3) * 2 + (q & 1);
                if (!third || m == 0) take_grad(g, o + e, ob + e, acc[i][t][q]);
            }
}

__global__ void to_bf16_kernel(const float *src, uint16_t *dst, long count)
{
    const long i = (long) blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= count) return;
    dst[i] = bf_bits(src[i]);
}

static unsigned blocks(long count, int t) { return (unsigned) ((count + t - 1) / t); }

// ---------------------------------------------------------------------------------------------

long Sifter::nparams() { return kNparams; }

Sifter::Sifter(int device_, long max_batch_, uint64_t seed) : device(device_), max_batch(max_batch_)
{
    if (max_batch < 1 || max_batch > 1024) throw std::runtime_error("Sifter: max_batch must be in [1, 1024]");
    SF_CHECK(cudaSetDevice(device));
    SF_CHECK(cudaMalloc(&master, kNparams * sizeof(float)));
    SF_CHECK(cudaMalloc(&grad, kNparams * sizeof(float)));
    SF_CHECK(cudaMalloc(&adam_m, kNparams * sizeof(float)));
    SF_CHECK(cudaMalloc(&adam_v, kNparams * sizeof(float)));
    SF_CHECK(cudaMalloc(&wb, kNbf16 * sizeof(uint16_t)));
    SF_CHECK(cudaMalloc(&z1, max_batch * kMlpH1 * sizeof(float)));
    SF_CHECK(cudaMalloc(&loss, sizeof(float)));
    SF_CHECK(cudaMalloc(&h1, max_batch * kMlpH1 * sizeof(uint16_t)));
    SF_CHECK(cudaMalloc(&h2, max_batch * kMlpH2 * sizeof(uint16_t)));
    SF_CHECK(cudaMalloc(&g, max_batch * sizeof(float)));
    SF_CHECK(cudaMalloc(&ls, max_batch * sizeof(float)));
    SF_CHECK(cudaMalloc(&g1, max_batch * kMlpH1 * sizeof(float)));
    SF_CHECK(cudaMalloc(&g2, max_batch * kMlpH2 * sizeof(float)));
    SF_CHECK(cudaMalloc(&gb, max_batch * kGPitch * sizeof(uint16_t)));
    SF_CHECK(cudaMalloc(&g1b, max_batch * kMlpH1 * sizeof(uint16_t)));
    SF_CHECK(cudaMalloc(&g2b, max_batch * kMlpH2 * sizeof(uint16_t)));
    SF_CHECK(cudaFuncSetAttribute(head_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) sizeof(HeadSmem)));
    SF_CHECK(cudaMemset(adam_m, 0, kNparams * sizeof(float)));
    SF_CHECK(cudaMemset(adam_v, 0, kNparams * sizeof(float)));
    // He-uniform initial weights, zero biases.
    std::vector<float> p(kNparams, 0.0f);
    std::mt19937_64 rng(seed);
    auto fill = [&](long off, long count, long fan_in) {
        std::uniform_real_distribution<double> u(-std::sqrt(6.0 / fan_in), std::sqrt(6.0 / fan_in));
        for (long i = 0; i < count; i++) p[off + i] = float(u(rng));
    };
    fill(oW1, kW1n, kMlpIn);
    fill(oW2, kW2n, kMlpH1);
    fill(oW3, kMlpH2, kMlpH2);
    set_params(p.data());
}

Sifter::~Sifter()
{
    cudaSetDevice(device);
    for (void *q : {(void *) master, (void *) grad, (void *) adam_m, (void *) adam_v, (void *) wb, (void *) z1,
                    (void *) loss, (void *) ls, (void *) h1, (void *) h2, (void *) g, (void *) g1, (void *) g2, (void *) gb,
                    (void *) g1b, (void *) g2b})
        if (q) cudaFree(q);
}

void Sifter::refresh_bf16(cudaStream_t s)
{
    to_bf16_kernel<<<blocks(kW1n, 256), 256, 0, s>>>(master + oW1, wb + bW1, kW1n);
    to_bf16_kernel<<<blocks(kW2n, 256), 256, 0, s>>>(master + oW2, wb + bW2, kW2n);
    to_bf16_kernel<<<blocks(kMlpH2, 256), 256, 0, s>>>(master + oW3, wb + bW3, kMlpH2);
    sf_check_launch("to_bf16_kernel");
}

void Sifter::set_params(const float *host)
{
    SF_CHECK(cudaSetDevice(device));
    SF_CHECK(cudaMemcpy(master, host, kNparams * sizeof(float), cudaMemcpyHostToDevice));
    refresh_bf16(nullptr);
    SF_CHECK(cudaDeviceSynchronize());
}

void Sifter::get_params(float *host) const
{
    SF_CHECK(cudaSetDevice(device));
    SF_CHECK(cudaMemcpy(host, master, kNparams * sizeof(float), cudaMemcpyDeviceToHost));
}

void Sifter::layer1(const uint16_t *patches, long n, cudaStream_t s)
{
    Layer1Args a;
    a.x = patches;
    a.w = wb + bW1;
    a.bias = master + oB1;
    a.n = int(n);
    a.aligned = (reinterpret_cast<uintptr_t>(patches) & 15) == 0;   // a patch is 3456 bytes
    a.z = z1;
    a.h = h1;
    layer1_kernel<<<dim3(kMlpH1 / 32, blocks(n, 32)), 128, 0, s>>>(a);
    sf_check_launch("layer1_kernel");
}

void Sifter::forward(const uint16_t *patches, long n, float *logits, cudaStream_t s)
{
    if (n < 1 || n > max_batch) throw std::runtime_error("Sifter::forward: batch size out of range");
    if (!patches || !logits) throw std::runtime_error("Sifter::forward: null pointer");
    layer1(patches, n, s);
    head(n, logits, nullptr, s);
}

// Layers 2 and 3 of the batch in h1: the logits, or with labels the loss terms and the gradients of the logits, Z2 and Z1.
void Sifter::head(long n, float *logits, const float *labels, cudaStream_t s)
{
    HeadArgs a;
    a.h1 = h1;
    a.w2 = wb + bW2;
    a.w3 = wb + bW3;
    a.z1 = z1;
    a.b2 = master + oB2;
    a.b3 = master + oB3;
    a.n = int(n);
    a.logits = logits;
    a.labels = labels;
    a.g = g;
    a.g2 = g2;
    a.g1 = g1;
    a.ls = ls;
    a.gb = gb;
    a.g2b = g2b;
    a.g1b = g1b;
    a.h2 = h2;
    head_kernel<<<blocks(n, kHeadRows), 256, sizeof(HeadSmem), s>>>(a);
    sf_check_launch("head_kernel");
}

// Forward and backward of the mean binary cross-entropy: the gradients into 'grad', or one Adam step.
void Sifter::train(const uint16_t *patches, const float *labels, long n, bool adam, float lr, cudaStream_t s)
{
    if (n < 1 || n > max_batch) throw std::runtime_error("Sifter::forward: batch size out of range");
    if (!patches) throw std::runtime_error("Sifter::forward: null pointer");
    layer1(patches, n, s);
    head(n, nullptr, labels, s);
    WgradArgs a;
    a.g1b = g1b;
    a.g2b = g2b;
    a.gb = gb;
    a.h1 = h1;
    a.h2 = h2;
    a.x = patches;
    a.g1 = g1;
    a.g2 = g2;
    a.g = g;
    a.ls = ls;
    a.n = int(n);
    a.aligned = (reinterpret_cast<uintptr_t>(patches) & 15) == 0;
    a.loss = loss;
    a.grad = adam ? nullptr : grad;
    a.w = master;
    a.m = adam_m;
    a.v = adam_v;
    a.wb = wb;
    a.lr = lr;
    a.c1 = 1.0f - std::pow(0.9f, float(step));
    a.c2 = 1.0f - std::pow(0.999f, float(step));
    wgrad_kernel<<<kWgTiles + kWgBias, 128, 0, s>>>(a);
    sf_check_launch("wgrad_kernel");
}

double Sifter::gradients(const uint16_t *patches, const float *labels, long n, float *grad_host, cudaStream_t s)
{
    if (!labels || !grad_host) throw std::runtime_error("Sifter::gradients: null pointer");
    SF_CHECK(cudaSetDevice(device));
    train(patches, labels, n, false, 0.0f, s);
    float l = 0.0f;
    SF_CHECK(cudaMemcpyAsync(grad_host, grad, kNparams * sizeof(float), cudaMemcpyDeviceToHost, s));
    SF_CHECK(cudaMemcpyAsync(&l, loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    SF_CHECK(cudaStreamSynchronize(s));
    return l;
}

double Sifter::train_step(const uint16_t *patches, const float *labels, long n, float lr, cudaStream_t s)
{
    if (!labels) throw std::runtime_error("Sifter::train_step: null pointer");
    SF_CHECK(cudaSetDevice(device));
    if (n >= 1 && n <= max_batch && patches) step++;
    train(patches, labels, n, true, lr, s);
    float l = 0.0f;
    SF_CHECK(cudaMemcpyAsync(&l, loss, sizeof(float), cudaMemcpyDeviceToHost, s));
    SF_CHECK(cudaStreamSynchronize(s));
    return l;
}

}  // namespace pb2
