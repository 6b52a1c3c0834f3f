// kernels.cu -- sm_100a kernels of the B200 dedispersion path.
//
//   grid_lds_kernel  tree gridding + lagged downsampling (replaces GpuTreeGriddingKernel,
//                    src_lib/TreeGriddingKernel.cu:108-279, and GpuLaggedDownsamplingKernel,
//                    src_lib/GpuLaggedDownsamplingKernel.cu:668-918)
//   pf_kernel      peak finding, max/argmax      (replaces the pf half of CoalescedDdKernel2 / GpuPeakFindingKernel)
//
// All arithmetic is fp32 in registers with explicit round-to-nearest intrinsics (no FMA contraction),
// performing the same sequence of fp32 operations as the reference CPU dedisperser, so that a float32
// plan reproduces its outputs bit for bit. Storage (inputs, tree intermediates, delay lines,
// out_max) is float32, float16 or bfloat16.

#include "kernels.cuh"
#include "devutil.cuh"

#include <cooperative_groups.h>
#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <string>
#include <type_traits>

namespace pb2 {

// Two fp32 additions (multiplications) in one sm_100 packed f32x2 instruction; each element is
// rounded to nearest like __fadd_rn (__fmul_rn).
__device__ __forceinline__ unsigned long long f2pack(float2 a)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 f2unpack(unsigned long long r)
{
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(r));
    return d;
}
__device__ __forceinline__ float2 f2add(float2 a, float2 b)
{
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f2pack(a)), "l"(f2pack(b)));
    return f2unpack(d);
}
__device__ __forceinline__ float2 f2mul(float2 a, float2 b)
{
    unsigned long long d;
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f2pack(a)), "l"(f2pack(b)));
    return f2unpack(d);
}

// -------------------------------------------------------------------------------------------------
// Tree gridding fused with lagged downsampling.
//
// Gridding: tree channel n = sum_f w[n,f] in[f], summed in ascending f from zero with float(w)
// overlap weights (ReferenceTreeGriddingKernel::apply, src_lib/TreeGriddingKernel.cu:62-102).
// Lagged downsampling, for each level p = 1..nlev:
//   ds_p[ch][u]  = (ds_{p-1}[ch][2u] + ds_{p-1}[ch][2u+1]) / sqrt2          (ds_0 = level-0 tree)
//   out_p[c][u]  = (ds_p[2c][u-1] + ds_p[2c+1][u]) / sqrt2                     (one-sample lag on even channels)
// out_p goes to a per-row delay line, written delayed by the per-row "large" lag
// 2^s1dd - 1 - (c mod 2^s1dd) (ReferenceLaggedDownsamplingKernel.cpp:46-57), so that the stage-1
// kernel reads aligned rows.
//
// One thread per (beam, tree-channel pair (2c, 2c+1), window of W0 level-0 samples); consecutive
// threads take consecutive windows, so every load and store is a contiguous run across the warp.
// The thread grids both channels of its window (and writes them as the level-0 tree), builds every
// level in registers, and gets the even channel's predecessor sample at each level by gridding the
// 2^nlev samples before its window (at the chunk start: from a parity double-buffered state).


// Loads W consecutive samples starting at p (16-byte vectors when W*sizeof(Ts) allows; p must then be
// 16-byte aligned).
template<typename Ts, int W>
__device__ __forceinline__ void load_run(const Ts *p, float (&o)[W])
{
    if constexpr ((W * sizeof(Ts)) % 16 == 0) {
        constexpr int PER = 16 / sizeof(Ts);
#pragma unroll
        for (int v = 0; v < W / PER; v++) {
            uint4 q = ((const uint4 *) p)[v];
            const Ts *h = (const Ts *) &q;
#pragma unroll
            for (int k = 0; k < PER; k++) o[v * PER + k] = to_f(h[k]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < W; i++) o[i] = to_f(p[i]);
    }
}

template<typename Ts, int W>
__device__ __forceinline__ void store_run(Ts *p, const float (&o)[W])
{
    if constexpr ((W * sizeof(Ts)) % 16 == 0) {
        constexpr int PER = 16 / sizeof(Ts);
#pragma unroll
        for (int v = 0; v < W / PER; v++) {
            uint4 q;
            Ts *h = (Ts *) &q;
#pragma unroll
            for (int k = 0; k < PER; k++) h[k] = from_f<Ts>(o[v * PER + k]);
            ((uint4 *) p)[v] = q;
        }
    } else {
#pragma unroll
        for (int i = 0; i < W; i++) p[i] = from_f<Ts>(o[i]);
    }
}

// int4 dequantization, restating pirate's ReferenceDequantizationKernel::apply
// (src_lib/GpuDequantizationKernel.cu:326-380): nibble -> signed value v in [-8, 7]; v = -8 is the
// "missing sample" sentinel and gives 0; otherwise scale * v + offset, one fp32 multiply and one fp32
// add with (scale, offset) converted from fp16. The result is then rounded once to the output type.
__device__ __forceinline__ float dq_value(uint32_t nib, float scale, float offset)
{
    // u = v + 8 in [0, 15]; 2^23 + u is exact in fp32, so subtracting 2^23 + 8 gives v exactly.
    const uint32_t u = (nib & 0xf) ^ 8u;
    const float fv = __fsub_rn(__uint_as_float(0x4B000000u + u), 8388616.0f);
    return (u == 0) ? 0.0f : __fadd_rn(__fmul_rn(scale, fv), offset);
}

// W consecutive samples from t0 of one int4 row (row = the row's bytes, so = its (scale, offset)
// pairs), dequantized, rounded to Ts and returned as floats. The W samples lie in one 256-sample
// scale block; for W >= 8, t0 is a multiple of 8 (32-bit nibble words).
template<typename Ts, int W>
__device__ __forceinline__ void load_run_q(const uint8_t *row, const __half2 *so_row, long t0, float (&o)[W])
{
    const float2 so = __half22float2(so_row[t0 >> 8]);
    if constexpr (W % 8 == 0) {
#pragma unroll
        for (int w = 0; w < W / 8; w++) {
            const uint32_t word = ((const uint32_t *) (row + (t0 >> 1)))[w];
#pragma unroll
            for (int k = 0; k < 8; k++) o[8 * w + k] = to_f(from_f<Ts>(dq_value(word >> (4 * k), so.x, so.y)));
        }
    } else {
#pragma unroll
        for (int i = 0; i < W; i++) {
            const long t = t0 + i;
            const uint32_t byte = row[t >> 1];
            o[i] = to_f(from_f<Ts>(dq_value((t & 1) ? (byte >> 4) : byte, so.x, so.y)));
        }
    }
}

// Grids tree channel n over samples [t0, t0+W) of batch beam b's input. With Q the input rows are
// int4 (dequantized on load exactly as the standalone dequantization kernel would write them).
template<typename Ts, int W, bool Q>
__device__ __forceinline__ void grid_run(const GridLdsArgs &a, int b, long n, long t0, float (&o)[W])
{
#pragma unroll
    for (int i = 0; i < W; i++) o[i] = 0.0f;
    const int f0 = a.chan_f0[n], cnt = a.chan_cnt[n], woff = a.chan_woff[n];
    for (int k = 0; k < cnt; k++) {
        const float w = a.chan_w[woff + k];
        const long row = (long) b * a.F + f0 + k;
        float x[W];
        if constexpr (Q)
            load_run_q<Ts, W>((const uint8_t *) a.q_data + row * (a.T >> 1), (const __half2 *) a.q_scoff + row * (a.T >> 8), t0, x);
        else
            load_run<Ts, W>((const Ts *) a.in + row * a.T + t0, x);
#pragma unroll
        for (int i = 0; i < W; i++) o[i] = __fadd_rn(o[i], __fmul_rn(w, x[i]));
    }
}

// int4 gridding through per-warp lookup tables. A warp's 32 windows of one tree-channel pair read the
// same few input rows, each input sample once per tree channel that overlaps its row (about 2.5 times
// at rank 16 from 16384 channels). Instead of dequantizing on every read, the warp first tabulates,
// per (row, 256-sample scale block), the 16 values its nibbles can take, rounded to Ts exactly as
// load_run_q rounds them; each read is then a nibble extract and a shared-memory lookup.
constexpr int kLutRows = 8;   // input rows per channel pair served by the tables

// Table of the warp: lut[(r * NBLK + blk) * 16 + u] = sample value of nibble u in row rlo + r, scale
// block blk0 + blk.
template<typename Ts, int NBLK>
__device__ __forceinline__ void lut_build(const GridLdsArgs &a, int b, int rlo, int nrows, long blk0, float *lut, int lane)
{
    const __half2 *so = (const __half2 *) a.q_scoff;
    const long nsb = a.T >> 8;
    for (int e = lane; e < nrows * NBLK * 16; e += 32) {
        const int r = e / (NBLK * 16), blk = (e / 16) % NBLK, u = e & 15;
        const float2 sc = __half22float2(so[((long) b * a.F + rlo + r) * nsb + blk0 + blk]);
        lut[e] = to_f(from_f<Ts>(dq_value(uint32_t(u), sc.x, sc.y)));
    }
    __syncwarp();
}

// The nibble words of a window of W samples (W / 8 words) of input row 'row' (t0 a multiple of 8).
template<int W>
__device__ __forceinline__ void lut_words(const GridLdsArgs &a, long row, long t0, uint32_t (&q)[W / 8])
{
    const uint32_t *p = (const uint32_t *) ((const uint8_t *) a.q_data + row * (a.T >> 1) + (t0 >> 1));
#pragma unroll
    for (int v = 0; v < W / 8; v++) q[v] = p[v];
}

// o += w * (row's samples), the samples looked up in table L.
template<int W>
__device__ __forceinline__ void lut_accum(float (&o)[W], float w, const uint32_t (&q)[W / 8], const float *L)
{
#pragma unroll
    for (int v = 0; v < W / 8; v++)
#pragma unroll
        for (int k8 = 0; k8 < 8; k8++) o[8 * v + k8] = __fadd_rn(o[8 * v + k8], __fmul_rn(w, L[(q[v] >> (4 * k8)) & 15]));
}

// grid_run<Ts, W, true> of tree channel n through the warp's tables (W a multiple of 8, t0 in scale
// block blk0 + myblk), summed in ascending input channel. q0 holds the words of the channel's first
// input row (loaded by the caller before the tables were built); later rows are loaded here.
template<typename Ts, int W, int NBLK>
__device__ __forceinline__ void grid_run_lut(const GridLdsArgs &a, int b, int f0, int cnt, int woff, long t0, float (&o)[W],
                                             const uint32_t (&q0)[W / 8], const float *lut, int rlo, int myblk)
{
#pragma unroll
    for (int i = 0; i < W; i++) o[i] = 0.0f;
    if (cnt > 0)
        lut_accum<W>(o, a.chan_w[woff], q0, lut + ((f0 - rlo) * NBLK + myblk) * 16);
    for (int k = 1; k < cnt; k++) {
        uint32_t q[W / 8];
        lut_words<W>(a, (long) b * a.F + f0 + k, t0, q);
        lut_accum<W>(o, a.chan_w[woff + k], q, lut + ((f0 + k - rlo) * NBLK + myblk) * 16);
    }
}

// Standalone dequantization, bound by HBM. A thread turns 16 output bytes' worth of samples at a time, so that a
// warp's loads and stores are each one contiguous run, four of them a block apart in flight. Rows are multiples of
// 256 samples and contiguous, so sample, scale block and byte offsets are the flat index's. (One thread per 32
// samples stored 16 bytes per lane 64 bytes apart: 81.7 us for 4 x 16384 x 2048 samples to fp16, against 67.5 us, 5.0 TB/s.)
constexpr int kDequantUnroll = 4;

template<typename To>
__global__ void __launch_bounds__(256) dequant_kernel(To *out, const uint8_t *data, const __half2 *scoff, long units)
{
    constexpr int SPT = 16 / sizeof(To);   // 4 or 8 samples
    using In = typename std::conditional<SPT == 8, uint32_t, uint16_t>::type;
    const long u0 = (long) blockIdx.x * (256 * kDequantUnroll) + threadIdx.x;
    In w[kDequantUnroll];
    float2 so[kDequantUnroll];
#pragma unroll
    for (int k = 0; k < kDequantUnroll; k++) {
        const long u = u0 + 256 * k;
        if (u < units) {
            w[k] = __ldg((const In *) data + u);
            so[k] = __half22float2(__ldg(scoff + (u * SPT >> 8)));
        }
    }
#pragma unroll
    for (int k = 0; k < kDequantUnroll; k++) {
        const long u = u0 + 256 * k;
        if (u < units) {
            float o[SPT];
#pragma unroll
            for (int i = 0; i < SPT; i++) o[i] = dq_value(uint32_t(w[k]) >> (4 * i), so[k].x, so[k].y);
            store_run<To, SPT>(out + u * SPT, o);
        }
    }
}

template<typename To>
static void launch_dequant_t(void *out, const void *data, const void *scoff, long samples, cudaStream_t s)
{
    const long units = samples / (16 / long(sizeof(To))), grid = (units + 256 * kDequantUnroll - 1) / (256 * kDequantUnroll);
    dequant_kernel<To><<<(unsigned) grid, 256, 0, s>>>((To *) out, (const uint8_t *) data, (const __half2 *) scoff, units);
}

void launch_dequantize(void *out, int out_dtype, const void *data, const void *scales_offsets, long nbeams, long nfreq,
                       long ntime, cudaStream_t s)
{
    if (ntime <= 0 || ntime % 256) throw std::runtime_error("dequantize: ntime must be a positive multiple of 256");
    if (!out || !data || !scales_offsets) throw std::runtime_error("dequantize: null pointer");
    const long samples = nbeams * nfreq * ntime;
    if (samples == 0) return;
    if (out_dtype == 0) launch_dequant_t<float>(out, data, scales_offsets, samples, s);
    else if (out_dtype == 1) launch_dequant_t<__half>(out, data, scales_offsets, samples, s);
    else launch_dequant_t<__nv_bfloat16>(out, data, scales_offsets, samples, s);
    check_launch("dequant_kernel");
}

// ---------------------------------------------------------------------------------------------
// Per-beam peak over a batch's outputs (the toy grouper's reduction, see BeamPeakArgs). The blocks of one cluster
// share a beam: each scans its slice of every tree with 16-byte loads where the beam's data is aligned, keeping per
// thread the largest value and its first index, and reduces them per tree; the first block then merges the slices
// through distributed shared memory and the trees in order. One block per beam left the chip to as many SMs as
// beams: 8 beams of a rank-16 plan (12.3 MB) took 44.7 us a call against 25.2 us, most of it the call's host part.

// Largest of the 16 bytes' elements (NaN if any is NaN), and element k, as fp32.
template<typename T> struct PeakVec;
template<> struct PeakVec<float>
{
    static constexpr int N = 4;
    __device__ static float max(const uint4 &q)
    {
        float m;
        asm("{.reg .f32 a, b;\n max.NaN.f32 a, %1, %2;\n max.NaN.f32 b, %3, %4;\n max.NaN.f32 %0, a, b;}"
            : "=f"(m) : "f"(__uint_as_float(q.x)), "f"(__uint_as_float(q.y)), "f"(__uint_as_float(q.z)), "f"(__uint_as_float(q.w)));
        return m;
    }
    __device__ static float get(const uint4 &q, int k) { return __uint_as_float(k == 0 ? q.x : k == 1 ? q.y : k == 2 ? q.z : q.w); }
};
template<> struct PeakVec<__half>
{
    static constexpr int N = 8;
    __device__ static float max(const uint4 &q)
    {
        const __half2 m = __hmax2_nan(__hmax2_nan(*(const __half2 *) &q.x, *(const __half2 *) &q.y),
                                      __hmax2_nan(*(const __half2 *) &q.z, *(const __half2 *) &q.w));
        return __half2float(__hmax_nan(__low2half(m), __high2half(m)));
    }
    __device__ static float get(const uint4 &q, int k)
    {
        const uint32_t w = (k < 2) ? q.x : (k < 4) ? q.y : (k < 6) ? q.z : q.w;
        return __half2float(__ushort_as_half((unsigned short) ((k & 1) ? (w >> 16) : (w & 0xffff))));
    }
};
template<> struct PeakVec<__nv_bfloat16>
{
    static constexpr int N = 8;
    __device__ static float max(const uint4 &q)
    {
        const __nv_bfloat162 m = __hmax2_nan(__hmax2_nan(*(const __nv_bfloat162 *) &q.x, *(const __nv_bfloat162 *) &q.y),
                                             __hmax2_nan(*(const __nv_bfloat162 *) &q.z, *(const __nv_bfloat162 *) &q.w));
        return __bfloat162float(__hmax_nan(__low2bfloat16(m), __high2bfloat16(m)));
    }
    __device__ static float get(const uint4 &q, int k)
    {
        const uint32_t w = (k < 2) ? q.x : (k < 4) ? q.y : (k < 6) ? q.z : q.w;
        return __uint_as_float((k & 1) ? (w & 0xffff0000u) : (w << 16));
    }
};

// A slice's maximum and its first index; v is NaN where the slice holds a NaN.
struct PeakPart
{
    float v;
    int i;
};
constexpr int kPeakNone = 0x7fffffff;

// The larger, on a tie the smaller index; NaN if either is.
__device__ __forceinline__ PeakPart peak_merge(PeakPart a, PeakPart b)
{
    if (a.v != a.v) return a;
    if (b.v != b.v) return b;
    return (b.v > a.v || (b.v == a.v && b.i < a.i)) ? b : a;
}

__device__ __forceinline__ PeakPart peak_warp(PeakPart p)
{
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        PeakPart q;
        q.v = __shfl_xor_sync(0xffffffffu, p.v, o);
        q.i = __shfl_xor_sync(0xffffffffu, p.i, o);
        p = peak_merge(p, q);
    }
    return p;
}

template<typename T>
__global__ void __launch_bounds__(1024) beam_peak_kernel(BeamPeakArgs a)
{
    namespace cg = cooperative_groups;
    cg::cluster_group cl = cg::this_cluster();
    constexpr int V = PeakVec<T>::N;
    __shared__ PeakPart wp[kBeamPeakMaxTrees][32];   // per tree and warp; in the first block, per tree the merged slices
    __shared__ PeakPart bp[kBeamPeakMaxTrees];       // per tree, this block's slice
    const int C = int(cl.num_blocks()), rank = int(cl.block_rank());
    const int b = blockIdx.x / C, lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    const int nwarps = blockDim.x >> 5;

    for (int t = 0; t < a.ntrees; t++) {
        const long n = a.ndm[t] * a.nt[t];
        const T *x = (const T *) a.out_max[t] + (long) b * n;
        PeakPart p = {-INFINITY, kPeakNone};
        bool nan = false;
        if (n % V == 0 && ((uintptr_t) x & 15) == 0) {
            const long nv = n / V, per = (nv + C - 1) / C;
            const long lo = rank * per, hi = min(nv, lo + per);
            const uint4 *xv = (const uint4 *) x;
            for (long j = lo + threadIdx.x; j < hi; j += 4L * blockDim.x) {
                uint4 q[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const long jj = j + (long) u * blockDim.x;
                    if (jj < hi) q[u] = __ldg(xv + jj);
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const long jj = j + (long) u * blockDim.x;
                    if (jj < hi) {
                        const float m = PeakVec<T>::max(q[u]);
                        nan |= (m != m);
                        if (m > p.v) {
                            p.v = m;
#pragma unroll
                            for (int k = V - 1; k >= 0; k--)
                                if (PeakVec<T>::get(q[u], k) == m) p.i = int(jj * V) + k;
                        }
                    }
                }
            }
        } else {
            const long per = (n + C - 1) / C, lo = rank * per, hi = min(n, lo + per);
            for (long i = lo + threadIdx.x; i < hi; i += blockDim.x) {
                const float v = to_f(x[i]);
                nan |= (v != v);
                if (v > p.v) { p.v = v; p.i = int(i); }
            }
        }
        if (nan) p.v = NAN;
        p = peak_warp(p);
        if (lane == 0) wp[t][warp] = p;
    }
    __syncthreads();
    for (int t = warp; t < a.ntrees; t += nwarps) {
        PeakPart p = {-INFINITY, kPeakNone};
        if (lane < nwarps) p = wp[t][lane];
        p = peak_warp(p);
        if (lane == 0) bp[t] = p;
    }
    cl.sync();
    if (rank == 0) {
        for (int t = warp; t < a.ntrees; t += nwarps) {
            PeakPart p = {-INFINITY, kPeakNone};
            if (lane < C) p = cl.map_shared_rank(bp, lane)[t];
            p = peak_warp(p);
            if (lane == 0) wp[t][0] = p;
        }
    }
    cl.sync();   // every slice has been read
    if (rank == 0 && threadIdx.x == 0) {
        // The first tree with the strictly largest maximum; a tree holding a NaN is passed over.
        float gv = -INFINITY;
        int gt = -1, gi = 0;
        for (int t = 0; t < a.ntrees; t++)
            if (wp[t][0].v > gv) { gv = wp[t][0].v; gt = t; gi = wp[t][0].i; }
        a.peak[b] = gv;
        a.tree[b] = gt;
        if (gt >= 0) {
            const long nt = a.nt[gt];
            a.idm[b] = int(gi / nt);
            a.itime[b] = int(gi % nt);
            a.token[b] = a.out_argmax[gt][(long) b * a.ndm[gt] * nt + gi];
        } else {
            a.idm[b] = -1;
            a.itime[b] = -1;
            a.token[b] = 0;
        }
    }
}

void launch_beam_peaks(const BeamPeakArgs &a, int dtype, long nbeams, cudaStream_t s)
{
    if (a.ntrees < 0 || a.ntrees > kBeamPeakMaxTrees) throw std::runtime_error("beam_peaks: bad number of trees");
    if (!a.peak || !a.tree || !a.idm || !a.itime || !a.token) throw std::runtime_error("beam_peaks: null output pointer");
    for (int t = 0; t < a.ntrees; t++) {
        if (!a.out_max[t] || !a.out_argmax[t]) throw std::runtime_error("beam_peaks: null output array");
        if (a.ndm[t] <= 0 || a.nt[t] <= 0 || a.ndm[t] * a.nt[t] >= (1L << 31))
            throw std::runtime_error("beam_peaks: tree shape out of range");
    }
    if (nbeams <= 0) return;
    if (nbeams > 0x7fffffffL) throw std::runtime_error("beam_peaks: too many beams");
    // Blocks per beam: up to 8 (the portable cluster size), about two per SM over all beams.
    unsigned C = 8;
    while (C > 1 && nbeams * C > 2 * 148) C /= 2;
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) nbeams * C);
    cfg.blockDim = dim3(1024);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = C;
    at[0].val.clusterDim.y = 1;
    at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    cudaError_t e;
    if (dtype == 0) e = cudaLaunchKernelEx(&cfg, beam_peak_kernel<float>, a);
    else if (dtype == 1) e = cudaLaunchKernelEx(&cfg, beam_peak_kernel<__half>, a);
    else if (dtype == 2) e = cudaLaunchKernelEx(&cfg, beam_peak_kernel<__nv_bfloat16>, a);
    else throw std::runtime_error("beam_peaks: dtype must be 0 (float32), 1 (float16) or 2 (bfloat16)");
    if (e != cudaSuccess) throw std::runtime_error(std::string("beam_peak_kernel: ") + cudaGetErrorString(e));
}

// ---------------------------------------------------------------------------------------------
// Pulse injection into a chunk (see launch_pulse_inject): one warp per channel, in the storage
// dtype, as out = round(out + weight * value) with one fp32 multiply and one fp32 add.

template<typename T>
__global__ void pulse_inject_kernel(T *out, long nfreq, long nt, long row_stride, long chunk_it0, const long *it0,
                                    const long *cnt, const long *off, const float *data, float weight)
{
    const long f = (long) blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5);
    if (f >= nfreq) return;
    const long a = it0[f] - chunk_it0;
    const long jlo = (a < 0) ? -a : 0;
    const long jhi = (cnt[f] < nt - a) ? cnt[f] : nt - a;
    const float *src = data + off[f];
    T *row = out + f * row_stride + a;
    for (long j = jlo + (threadIdx.x & 31); j < jhi; j += 32)
        row[j] = from_f<T>(__fadd_rn(to_f(row[j]), __fmul_rn(weight, src[j])));
}

void launch_pulse_inject(void *out, int dtype, long nfreq, long nt, long row_stride, long chunk_it0, const long *it0,
                         const long *cnt, const long *off, const float *data, float weight, cudaStream_t s)
{
    if (!out || !it0 || !cnt || !off || !data) throw std::runtime_error("pulse_inject: null pointer");
    if (nfreq <= 0 || nt <= 0 || row_stride < nt) throw std::runtime_error("pulse_inject: bad chunk shape");
    const unsigned grid = (unsigned) ((nfreq + 7) / 8);
    if (dtype == 0) pulse_inject_kernel<float><<<grid, 256, 0, s>>>((float *) out, nfreq, nt, row_stride, chunk_it0, it0, cnt, off, data, weight);
    else if (dtype == 1) pulse_inject_kernel<__half><<<grid, 256, 0, s>>>((__half *) out, nfreq, nt, row_stride, chunk_it0, it0, cnt, off, data, weight);
    else if (dtype == 2) pulse_inject_kernel<__nv_bfloat16><<<grid, 256, 0, s>>>((__nv_bfloat16 *) out, nfreq, nt, row_stride, chunk_it0, it0, cnt, off, data, weight);
    else throw std::runtime_error("pulse_inject: dtype must be 0 (float32), 1 (float16) or 2 (bfloat16)");
    check_launch("pulse_inject_kernel");
}

// ---------------------------------------------------------------------------------------------
// Host spill copies (see SpillArgs): one warp per (beam, spilled row), 16-byte vectors (a chunk row is
// nt * esize bytes, a multiple of 64; every offset is a multiple of 32 samples).

__device__ __forceinline__ long spill_mod(long x, long m) { long r = x % m; return r < 0 ? r + m : r; }

template<bool G2H>
__global__ void __launch_bounds__(256) spill_kernel(SpillArgs a)
{
    const long w = (long) blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (w >= (long) a.nrows * a.B) return;
    const int j = int(w % a.nrows), b = int(w / a.nrows), bt = a.beam0 + b;
    const SpillRow r = a.rows[j];
    const long c = a.chunk_ctr ? *a.chunk_ctr : a.ichunk;
    const long q = G2H ? c : c - r.d + 1;   // chunk moved this step
    const long slot = spill_mod(q, r.S);
    char *dev = (char *) a.ring + ((long) bt * a.ring_beam_stride + (G2H ? r.w_off : r.r_off + spill_mod(q, 2) * a.nt)) * a.esize;
    char *host = (char *) a.host + (r.h_base + ((slot * a.total_beams + bt) * r.n_z + r.k) * (long) a.nt) * a.esize;
    const int nv = a.nt * a.esize / 16;
    const uint4 *src = (const uint4 *) (G2H ? dev : host);
    uint4 *dst = (uint4 *) (G2H ? host : dev);
    for (int i = lane; i < nv; i += 32) dst[i] = src[i];
}

static void launch_spill(const SpillArgs &a, bool g2h, cudaStream_t s)
{
    if (a.nrows <= 0 || a.B <= 0) return;
    if (!a.ring || !a.host || !a.rows) throw std::runtime_error("spill: null pointer");
    if ((a.nt * a.esize) % 64) throw std::runtime_error("spill: chunk rows must be a multiple of 64 bytes");
    const long warps = (long) a.nrows * a.B;
    const unsigned grid = (unsigned) ((warps + 7) / 8);
    if (g2h) spill_kernel<true><<<grid, 256, 0, s>>>(a);
    else spill_kernel<false><<<grid, 256, 0, s>>>(a);
    check_launch("spill_kernel");
}

void launch_spill_g2h(const SpillArgs &a, cudaStream_t s) { launch_spill(a, true, s); }
void launch_spill_h2g(const SpillArgs &a, cudaStream_t s) { launch_spill(a, false, s); }

constexpr int kGridMaxThreads = 512;

template<typename Ts, int NLEV, bool Q>
__global__ void __launch_bounds__(kGridMaxThreads) grid_lds_kernel(GridLdsArgs a)
{
    constexpr int W0 = ((1 << NLEV) > 8) ? (1 << NLEV) : 8;
    constexpr int WE = 1 << NLEV;           // level-0 samples feeding one level-NLEV sample
    __shared__ float xch[(NLEV > 0) ? NLEV : 1][kGridMaxThreads];
    // int4 lookup tables (grid_run_lut): for windows of at most 16 samples, NBLK scale blocks per warp.
    constexpr bool LUT = Q && (W0 <= 16);
    constexpr int NBLK = LUT ? (32 * W0) / 256 : 1;
    __shared__ float lut_sh[LUT ? (kGridMaxThreads / 32) * kLutRows * NBLK * 16 : 1];

    const long nhalf = 1L << (a.rank - 1);
    const long nwin = a.T / W0;
    const long g = (long) blockIdx.x * blockDim.x + threadIdx.x;
    // Threads past the end take part in the block barrier only.
    const bool live = g < nwin * nhalf * a.B;
    const long gg = live ? g : 0;
    const int win = int(gg % nwin);
    const long c = (gg / nwin) % nhalf;
    const int b = int(gg / (nwin * nhalf));
    const int bt = a.beam0 + b;
    const long ichunk = a.chunk_ctr ? *a.chunk_ctr : a.ichunk;
    const int parity = int(ichunk & 1);
    const long t0 = (long) win * W0;

    float r0[W0], r1[W0];
    // A warp uses the tables when its 32 threads are live windows of one channel pair (nwin a multiple
    // of 32; blocks start at window 0) whose input rows fit; the choice is uniform across the warp.
    bool use_lut = false;
    if constexpr (LUT) {
        if (live && (nwin & 31) == 0) {
            const int fa = a.chan_f0[2 * c], ca = a.chan_cnt[2 * c], fb = a.chan_f0[2 * c + 1], cb = a.chan_cnt[2 * c + 1];
            const int rlo = min(ca ? fa : fb, cb ? fb : fa);
            const int rhi = max(fa + ca, fb + cb);
            use_lut = (rhi - rlo) <= kLutRows;
            if (use_lut) {
                // The first input row of each channel is loaded before the tables are built, so that its
                // latency overlaps that of the (scale, offset) loads.
                uint32_t qa[W0 / 8], qb[W0 / 8];
                lut_words<W0>(a, (long) b * a.F + (ca ? fa : rlo), t0, qa);
                lut_words<W0>(a, (long) b * a.F + (cb ? fb : rlo), t0, qb);
                const int wa = a.chan_woff[2 * c], wb = a.chan_woff[2 * c + 1];
                const int lane = threadIdx.x & 31;
                const long blk0 = ((long) (win - lane) * W0) >> 8;
                float *lut = lut_sh + (threadIdx.x >> 5) * (kLutRows * NBLK * 16);
                lut_build<Ts, NBLK>(a, b, rlo, rhi - rlo, blk0, lut, lane);
                const int myblk = int((t0 >> 8) - blk0);
                grid_run_lut<Ts, W0, NBLK>(a, b, fa, ca, wa, t0, r0, qa, lut, rlo, myblk);
                grid_run_lut<Ts, W0, NBLK>(a, b, fb, cb, wb, t0, r1, qb, lut, rlo, myblk);
            }
        }
    }
    if (live && !use_lut) {
        grid_run<Ts, W0, Q>(a, b, 2 * c, t0, r0);
        grid_run<Ts, W0, Q>(a, b, 2 * c + 1, t0, r1);
    }
    if (live) {
        Ts *lev0 = (Ts *) a.tree0 + ((long) b * (2 * nhalf) + 2 * c) * a.T + t0;
        store_run<Ts, W0>(lev0, r0);
        store_run<Ts, W0>(lev0 + a.T, r1);
    }

    if constexpr (NLEV > 0) {
        // Level p of each channel: in place, r[u] = (r[2u] + r[2u+1]) / sqrt2. The odd channel's output
        // sample u pairs with the even channel's sample u-1; for u = 0 that is the last sample of the
        // previous window at this level (the thread before, exchanged through shared memory), or at
        // the chunk start the saved state.
        float first[NLEV], last[NLEV];
#pragma unroll
        for (int p = 1; p <= NLEV; p++) {
            const int len = W0 >> p;
#pragma unroll
            for (int u = 0; u < (W0 >> 1); u++) {
                if (u < len) {
                    r0[u] = bfly(r0[2 * u], r0[2 * u + 1]);
                    r1[u] = bfly(r1[2 * u], r1[2 * u + 1]);
                }
            }
            first[p - 1] = r1[0];
            last[p - 1] = r0[len - 1];
            xch[p - 1][threadIdx.x] = r0[len - 1];

            if (live) {
                const long cap = a.cap_mask[p - 1] + 1;
                Ts *ring = (Ts *) a.ring[p - 1] + ((long) bt * nhalf + c) * cap;
                const long nt_p = a.T >> p;
                const long s_base = ichunk * nt_p + (long) win * len + ((1L << a.lag_rank) - 1 - (c & ((1L << a.lag_rank) - 1)));
#pragma unroll
                for (int u = 1; u < (W0 >> 1); u++)
                    if (u < len)
                        ring[(s_base + u) & a.cap_mask[p - 1]] = from_f<Ts>(bfly(r0[u - 1], r1[u]));
                if (win == nwin - 1)
                    a.state[(((long) (1 - parity) * a.total_beams + bt) * a.nlev + (p - 1)) * nhalf + c] = last[p - 1];
            }
        }
        __syncthreads();

        if (live) {
            float prev[NLEV];
            if (win == 0) {
#pragma unroll
                for (int p = 1; p <= NLEV; p++)
                    prev[p - 1] = a.state[(((long) parity * a.total_beams + bt) * a.nlev + (p - 1)) * nhalf + c];
            } else if (threadIdx.x > 0) {
#pragma unroll
                for (int p = 1; p <= NLEV; p++)
                    prev[p - 1] = xch[p - 1][threadIdx.x - 1];
            } else {
                // The previous window belongs to the previous block: grid its WE samples again.
                float e[WE];
                grid_run<Ts, WE, Q>(a, b, 2 * c, t0 - WE, e);
#pragma unroll
                for (int p = 1; p <= NLEV; p++) {
#pragma unroll
                    for (int u = 0; u < (WE >> 1); u++)
                        if (u < (WE >> p)) e[u] = bfly(e[2 * u], e[2 * u + 1]);
                    prev[p - 1] = e[(WE >> p) - 1];
                }
            }
#pragma unroll
            for (int p = 1; p <= NLEV; p++) {
                const long cap = a.cap_mask[p - 1] + 1;
                Ts *ring = (Ts *) a.ring[p - 1] + ((long) bt * nhalf + c) * cap;
                const long nt_p = a.T >> p;
                const long s_base = ichunk * nt_p + (long) win * (W0 >> p) + ((1L << a.lag_rank) - 1 - (c & ((1L << a.lag_rank) - 1)));
                ring[s_base & a.cap_mask[p - 1]] = from_f<Ts>(bfly(prev[p - 1], first[p - 1]));
            }
        }
    }
}


// -------------------------------------------------------------------------------------------------
// Peak finding. One warp per (beam, coarse dm, 32 consecutive output times). For each multiplet m
// the warp stages the input window in shared memory and builds the boxcar levels with the reference's
// recursion  B_{l+1}[u] = B_l[r u] + B_l[r u + s]  (so every boxcar sum has the reference's rounding);
// each lane then scans the trials of its output time. The running maximum breaks ties by the
// reference's scan order (level, multiplet, fine time, profile), reproducing its out_argmax tokens.


constexpr int kPfWarps = 4;
constexpr int kPfMaxLevels = 6;
constexpr int kPfMaxProfiles = 16;   // 1 + 3 log2(max_width), max_width <= 32

// Number of entries of boxcar level l in a window of len0 samples (level 0 = samples).
__device__ __forceinline__ int pf_nlev(int len0, int l, int dt) { return (len0 - (1 << l)) / dt + 1; }

template<typename Ts>
__device__ __forceinline__ float ld_f(const Ts *p) { return to_f(*p); }

// Loads multiplet row 'row' over the warp's window into lev[0..len0) and builds boxcar levels
// 1..L-1 after it with the reference recursion B_{l+1}[u] = B_l[r u] + B_l[r u + s].
template<typename Ts, int L>
__device__ __forceinline__ void pf_build(float *lev, int len0, int lane, int Dcore, const Ts *row, long s_base, long mask)
{
    for (int u = lane; u < len0; u += 32)
        lev[u] = to_f(row[(s_base + u) & mask]);
    __syncwarp();
    int off = 0;
#pragma unroll
    for (int l = 0; l + 1 < L; l++) {
        const int dt = min(Dcore, 1 << l), dt1 = min(Dcore, 1 << (l + 1));
        const int n = pf_nlev(len0, l, dt), n1 = pf_nlev(len0, l + 1, dt1);
        const int rr = dt1 / dt, ss = (1 << l) / dt;
        const float *src = lev + off;
        float *dst = lev + off + n;
        for (int u = lane; u < n1; u += 32)
            dst[u] = __fadd_rn(src[rr * u], src[rr * u + ss]);
        __syncwarp();
        off += n;
    }
}

// Group (level l, multiplet m) of one output time: the reference scans fine times 'is' and, per fine
// time, profiles p = 0 (level 0 only), 3l+1, 3l+2, 3l+3. Keeps the first maximum of the group.
template<bool P0>
__device__ __forceinline__ void pf_group(const float *x, int nsamp, int S, float w0, float w1, float w2, float w3,
                                         bool full, float &gmax, int &gidx)
{
    gmax = -1.0e30f;
    gidx = -1;
    if (S == 1) {
        float x0 = x[-3], x1 = x[-2], x2 = x[-1];
        for (int is = 0; is < nsamp; is++) {
            float x3 = x[is];
            if (P0) { float v = __fmul_rn(w0, x3); if (v > gmax) { gmax = v; gidx = 4 * is; } }
            if (full) {
                float hx3 = __fmul_rn(0.5f, x3);
                float v1 = __fmul_rn(w1, __fadd_rn(x2, x3));
                float v2 = __fmul_rn(w2, __fadd_rn(__fadd_rn(__fmul_rn(0.5f, x1), x2), hx3));
                float v3 = __fmul_rn(w3, __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(0.5f, x0), x1), x2), hx3));
                if (v1 > gmax) { gmax = v1; gidx = 4 * is + 1; }
                if (v2 > gmax) { gmax = v2; gidx = 4 * is + 2; }
                if (v3 > gmax) { gmax = v3; gidx = 4 * is + 3; }
            }
            x0 = x1; x1 = x2; x2 = x3;
        }
    } else {
        for (int is = 0; is < nsamp; is++) {
            float x0 = x[is - 3 * S], x1 = x[is - 2 * S], x2 = x[is - S], x3 = x[is];
            if (P0) { float v = __fmul_rn(w0, x3); if (v > gmax) { gmax = v; gidx = 4 * is; } }
            if (full) {
                float hx3 = __fmul_rn(0.5f, x3);
                float v1 = __fmul_rn(w1, __fadd_rn(x2, x3));
                float v2 = __fmul_rn(w2, __fadd_rn(__fadd_rn(__fmul_rn(0.5f, x1), x2), hx3));
                float v3 = __fmul_rn(w3, __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(0.5f, x0), x1), x2), hx3));
                if (v1 > gmax) { gmax = v1; gidx = 4 * is + 1; }
                if (v2 > gmax) { gmax = v2; gidx = 4 * is + 2; }
                if (v3 > gmax) { gmax = v3; gidx = 4 * is + 3; }
            }
        }
    }
}

// One warp per (beam, coarse dm, 32 consecutive output times). For each multiplet the warp stages
// the input window in shared memory and builds the boxcar levels (every boxcar sum has the
// reference's rounding); each lane then scans the trials of its output time. Across groups the
// winner is the first group, in the reference's scan order (level, multiplet), whose maximum equals
// the overall maximum; within a group the first trial reaching it. This reproduces
// ReferencePeakFindingKernel::apply's strict-'>' sequential scan (src_lib/PeakFindingKernel.cu:339-420).
template<typename Ts, int L>
__global__ void __launch_bounds__(kPfWarps * 32) pf_kernel(PfArgs a, int warp_floats)
{
    const long s0 = a.chunk_ctr ? *a.chunk_ctr * (long) a.nt_chunk : a.s0;
    extern __shared__ float sm[];
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const int dm = blockIdx.y * kPfWarps + warp;
    const int b = blockIdx.z, bt = a.beam0 + b;
    const int tout0 = blockIdx.x * 32;
    if (dm >= a.ndm_out)
        return;   // whole warp exits; warps never synchronize across the block

    const int ntw = min(32, a.nt_out - tout0);
    const int len0 = ntw * a.Dout + a.tpad;
    float *lev = sm + warp * warp_floats;

    const int tout = tout0 + lane;
    const bool active = (lane < ntw);
    const int Wds = a.ndm_out / a.ndm_wt, Tds = a.nt_out / a.nt_wt;
    const float *wp = a.wt + ((((long) b * a.ndm_wt + dm / Wds) * a.nt_wt + (active ? tout / Tds : 0)) * a.P) * a.N;
    const Ts *pfrows = (const Ts *) a.pf + ((long) bt * a.ndm_out + dm) * a.M * a.pf_cap;
    const long mask = a.pf_cap - 1;
    const long s_base = s0 + (long) tout0 * a.Dout - a.tpad;
    const bool full = (a.P > 1);

    float best = -1.0e30f;
    int win = 0x7fffffff;     // (l * M + m) * 256 + in-group index of the winning trial

    for (int m = 0; m < a.M; m++) {
        pf_build<Ts, L>(lev, len0, lane, a.Dcore, pfrows + (long) m * a.pf_cap, s_base, mask);
        if (active) {
            const int n = a.m_to_n[m];
            int off = 0;
#pragma unroll
            for (int l = 0; l < L; l++) {
                const int dt = min(a.Dcore, 1 << l), S = (1 << l) / dt, nsamp = a.Dout / dt;
                const int I = (a.tpad + dt - (1 << l)) / dt;
                const float *x = lev + off + I + lane * nsamp;
                float w0 = (l == 0) ? wp[n] : 0.0f, w1 = 0.0f, w2 = 0.0f, w3 = 0.0f;
                if (full) {
                    w1 = wp[(3 * l + 1) * a.N + n];
                    w2 = wp[(3 * l + 2) * a.N + n];
                    w3 = wp[(3 * l + 3) * a.N + n];
                }
                float gmax;
                int gidx;
                if (l == 0) pf_group<true>(x, nsamp, S, w0, w1, w2, w3, full, gmax, gidx);
                else pf_group<false>(x, nsamp, S, w0, w1, w2, w3, full, gmax, gidx);
                const int g = ((l * a.M + m) << 8) + gidx;
                if (gidx >= 0 && (gmax > best || (gmax == best && g < win))) { best = gmax; win = g; }
                off += pf_nlev(len0, l, dt);
            }
        }
        __syncwarp();
    }

    if (active) {
        uint32_t tok = 0xffffffffu;
        if (win != 0x7fffffff) {
            const int gi = win & 255, grp = win >> 8;
            const int l = grp / a.M, m = grp % a.M;
            const int dt = min(a.Dcore, 1 << l);
            const int is = gi >> 2, q = gi & 3;
            const int p = (q == 0) ? 0 : (3 * l + q);
            tok = (uint32_t(m) << 16) | (uint32_t(p) << 8) | uint32_t(is * dt);
        }
        long o = ((long) b * a.ndm_out + dm) * a.nt_out + tout;
        ((Ts *) a.out_max)[o] = from_f<Ts>(best);
        a.out_argmax[o] = tok;
    }
}


// -------------------------------------------------------------------------------------------------
// Fast peak finding (output time downsampling Dout >= 4; the general kernel above covers the rest).
//
// Same work split (one warp per beam, coarse dm and 32 output times; lane = output time) and the same
// results, organised around four changes:
//
//  1. Bank-conflict-free shared memory. Level l of the boxcar window is stored in blocks of nsamp_l
//     entries (one block per lane: its output time's fine samples). Levels scanned in pairs with
//     blocks of >= 4 entries pad each block with 2 floats, so the 32 blocks fall on distinct banks
//     for 8-byte loads; the other levels are contiguous and are read in pairs or single floats.
//  2. Levels are built while they are scanned: while a lane scans its fine samples at level l two at
//     a time, the pair's sum is its level-(l+1) entry (B_{l+1}[u] = B_l[2u] + B_l[2u+1] while
//     dt doubles), so only the pad region before the first output time and the levels with
//     saturated time step (dt = Dcore) are built in a separate pass.
//  3. Max-only trial loop. The scan keeps, per group (level, multiplet), the maximum trial value
//     (fmaxf and the three-input max, which ignore NaN as the reference's strict '>' does) and the
//     first fine sample (pair) reaching it; across groups, the first group in the reference's
//     (level, multiplet) order whose maximum equals the overall one. After each multiplet, a lane
//     whose maximum moved into it recomputes that fine sample's (pair's) trials from shared memory
//     and takes the first, in (fine time, profile) order, equal to the maximum: its value and token
//     are the outputs.
//  4. The next multiplet's window is staged in shared memory with cp.async while the current one is
//     scanned.

// Per-level constants of the fast peak finder (host-computed; level l has time step dt, boxcar
// length 2^l = S*dt, and nsamp = Dout/dt fine samples per output time).
enum { kPfU = 1, kPfPairs = 2, kPfNextU = 4 };
struct PfGeom
{
    int off[kPfMaxLevels];   // first float of level l in a warp's region (even)
    int e[kPfMaxLevels];     // entry i lies in block (i + e) >> k
    int k[kPfMaxLevels];     // log2(nsamp_l)
    int pad[kPfMaxLevels];   // floats after each block
    int I[kPfMaxLevels];     // entry of the warp's first output time's first fine sample
    int n[kPfMaxLevels];     // entries of level l in the window of 32 output times
    int dt[kPfMaxLevels], S[kPfMaxLevels], nsamp[kPfMaxLevels];
    int rr[kPfMaxLevels], ss[kPfMaxLevels];   // B_l[u] = B_{l-1}[rr u] + B_{l-1}[rr u + ss]
    int flags[kPfMaxLevels]; // kPfU: dt = 2^l; kPfPairs: scanned two fine samples at a time;
                             // kPfNextU: level l+1 has dt = 2^(l+1) and is built by this level's scan
    int raw_off;             // two staging buffers of the window's raw samples (16-byte aligned), one per
    int raw_floats;          // multiplet in flight, raw_floats apart; level 0 is read from them directly
    int w_off;               // the warp's weights of one subband, [profile < 16][weight time < 32]
    int warp_floats;
};

// max(a, b, c) ignoring NaN inputs (sm_100 three-input max).
__device__ __forceinline__ float pf_max3(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

__device__ __forceinline__ int pf_phys(const PfGeom &g, int l, int i)
{
    const int t = i + g.e[l];
    return g.off[l] + t + g.pad[l] * (t >> g.k[l]);
}

template<typename Ts> __device__ __forceinline__ void pf_load4(const Ts *p, float (&v)[4]);
template<> __device__ __forceinline__ void pf_load4<float>(const float *p, float (&v)[4])
{
    const float4 q = *(const float4 *) p;
    v[0] = q.x; v[1] = q.y; v[2] = q.z; v[3] = q.w;
}
template<> __device__ __forceinline__ void pf_load4<__half>(const __half *p, float (&v)[4])
{
    const uint2 q = *(const uint2 *) p;
    const float2 a = __half22float2(*(const __half2 *) &q.x), b = __half22float2(*(const __half2 *) &q.y);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
template<> __device__ __forceinline__ void pf_load4<__nv_bfloat16>(const __nv_bfloat16 *p, float (&v)[4])
{
    const uint2 q = *(const uint2 *) p;
    const float2 a = __bfloat1622float2(*(const __nv_bfloat162 *) &q.x), b = __bfloat1622float2(*(const __nv_bfloat162 *) &q.y);
    v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
}
// Eight samples from a 16-byte-aligned address (two 4-sample loads for fp32).
template<typename Ts> __device__ __forceinline__ void pf_load8(const Ts *p, float (&v)[8])
{
    if constexpr (sizeof(Ts) == 4) {
        float a[4], b[4];
        pf_load4<Ts>(p, a);
        pf_load4<Ts>(p + 4, b);
#pragma unroll
        for (int i = 0; i < 4; i++) { v[i] = a[i]; v[4 + i] = b[i]; }
    } else {
        const uint4 q = *(const uint4 *) p;
        const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
        for (int i = 0; i < 4; i++) {
            float2 f;
            if constexpr (std::is_same<Ts, __half>::value) f = __half22float2(*(const __half2 *) &w[i]);
            else f = __bfloat1622float2(*(const __nv_bfloat162 *) &w[i]);
            v[2 * i] = f.x; v[2 * i + 1] = f.y;
        }
    }
}

// Shared-memory layout of the fast peak finder for one warp (see PfGeom).
// LW: output times (lanes) per coarse DM in a warp (32, or 16 and 8 for trees with that few output
// times per chunk: 32 / LW coarse DMs then share a warp).
__host__ __device__ constexpr PfGeom pf_geom(int Dout, int Dcore, int tpad, int L, int esize, int LW = 32)
{
    PfGeom g{};
    int off = 0;
    for (int l = 0; l < L; l++) {
        const int dt = (Dcore < (1 << l)) ? Dcore : (1 << l);
        const int nsamp = Dout / dt;
        const bool pairs = ((1 << l) <= Dcore) && nsamp >= 2;
        const int I = (tpad + dt - (1 << l)) / dt;
        int k = 0;
        while ((1 << k) < nsamp) k++;
        g.off[l] = off;
        g.e[l] = (nsamp - I % nsamp) % nsamp;
        g.k[l] = k;
        // Levels scanned in pairs from per-lane blocks: 2 floats after each block of >= 4 (the
        // blocks then fall on distinct banks for 8-byte loads); the others are stored contiguously.
        g.pad[l] = (pairs && nsamp >= 4) ? 2 : 0;
        g.I[l] = I;
        g.n[l] = LW * nsamp + I;
        g.dt[l] = dt;
        g.S[l] = (1 << l) / dt;
        g.nsamp[l] = nsamp;
        if (l > 0) {
            const int dtp = (Dcore < (1 << (l - 1))) ? Dcore : (1 << (l - 1));
            g.rr[l] = dt / dtp;
            g.ss[l] = (1 << (l - 1)) / dtp;
        }
        g.flags[l] = (((1 << l) <= Dcore) ? kPfU : 0) | (pairs ? kPfPairs : 0)
                   | ((l + 1 < L && (2 << l) <= Dcore) ? kPfNextU : 0);
        const int t = g.n[l] - 1 + g.e[l];
        const int size = t + g.pad[l] * (t >> k) + 1;
        if (l > 0)   // level 0 lives only in the raw staging buffer
            off += (size + 1) & ~1;
    }
    g.raw_off = (off + 3) & ~3;
    g.raw_floats = ((LW * Dout + tpad) * esize + 15) / 16 * 4;
    g.w_off = g.raw_off + 2 * g.raw_floats;
    g.warp_floats = g.w_off + kPfMaxProfiles * 32;
    return g;
}

// Peak-finder constants fixed by the plan rules: Dcore = min(Dout, 8) and tpad = max(2 Wmax, 4) with
// L = max(log2 Wmax, 1), i.e. tpad = max(2^(L+1), 4).
__host__ __device__ constexpr int pf_dcore_of(int Dout) { return Dout < 8 ? Dout : 8; }
__host__ __device__ constexpr int pf_tpad_of(int L) { return (2 << L) > 4 ? (2 << L) : 4; }

// The kernel body. g holds the per-level constants (a compile-time constant object when DOUT > 0, so
// the unrolled level loop sees them as immediates); gr is the same geometry passed at launch, used
// where the level is only known at run time.
// CTR: the chunk index comes from the device counter (replayed CUDA graphs). It is a template flag
// because reading it costs the kernel about 26 registers, which the direct launches should not pay.
template<typename Ts, int L, int DOUT, bool CTR, int LW>
__device__ __forceinline__ void pf_fast_body(const PfArgs &a, const PfGeom &g, const PfGeom &gr)
{
    static_assert(LW == 32 || LW == 16 || LW == 8, "lanes per coarse DM");
    constexpr int G = 32 / LW;   // coarse DMs per warp, each on LW consecutive lanes
    extern __shared__ float sm[];
    const int warp = threadIdx.x >> 5, sub = (threadIdx.x & 31) / LW, lane = threadIdx.x & (LW - 1);
    const int dm0 = (blockIdx.y * kPfWarps + warp) * G;
    const int b = blockIdx.z, bt = a.beam0 + b;
    const int tout0 = blockIdx.x * LW;
    if (dm0 >= a.ndm_out)
        return;   // whole warp exits; warps never synchronize across the block
    // A sub-group past the last coarse DM computes the last one again and stores nothing.
    const bool dm_ok = dm0 + sub < a.ndm_out;
    const int dm = dm_ok ? dm0 + sub : a.ndm_out - 1;

    const int ntw = min(LW, a.nt_out - tout0);
    const int tout = tout0 + lane;
    const bool active = (lane < ntw) && dm_ok;
    float *lev = sm + (warp * G + sub) * g.warp_floats;

    const int Dout = (DOUT > 0) ? DOUT : a.Dout;
    const int tpad = (DOUT > 0) ? pf_tpad_of(L) : a.tpad;
    const int Wds = a.ndm_out / a.ndm_wt, Tds = a.nt_out / a.nt_wt;
    // Weights of one subband for the warp's weight times tw0 .. tw0 + NT - 1, staged in shared memory
    // as wsm[p * 32 + j] (lanes of one weight time read the same word, consecutive weight times
    // consecutive words), and reloaded only when a multiplet's subband differs from the previous one.
    const float *wrow = a.wt + ((long) b * a.ndm_wt + dm / Wds) * a.nt_wt * a.P * a.N;
    const int tw0 = tout0 / Tds, NT = (Tds >= LW) ? 1 : LW / Tds;
    const int tl = (lane < ntw) ? (tout / Tds - tw0) : 0;
    float *wsm = lev + g.w_off;
    int wsm_n = -1;
    const Ts *pfrows = (const Ts *) a.pf + ((long) bt * a.ndm_out + dm) * a.M * a.pf_cap;
    const int mask = int(a.pf_cap - 1);
    // Window sample 0 (stream time s0 + 32 tile * Dout - tpad, a multiple of 4), as a delay-line slot.
    long s0 = a.s0;
    if constexpr (CTR) s0 = *a.chunk_ctr * (long) a.nt_chunk;
    const int sbm = int((s0 + (long) tout0 * Dout - tpad) & (a.pf_cap - 1));
    const bool full = (L > 1) || (a.P > 1);
    const int nq0 = (ntw * Dout + tpad) >> 2;   // samples the active lanes read (a partial last tile reads fewer)

    float best = -1.0e30f;
    int winG = -1;            // group l * M + m of the first maximum; -1: no trial above -1e30
    float outv = best;        // value and token of the first maximal trial
    uint32_t tok = 0xffffffffu;
    // Inputs of the winning group's first maximal pair, saved when the maximum moves, so that the
    // token is found once at the end: x[j - 3S .. j] of its samples is = winP (a) and winP + 1 (b),
    // the level's weights, and the pair's level, multiplet and start.
    float xa0 = 0, xa1 = 0, xa2 = 0, xa3 = 0, xb0 = 0, xb1 = 0, xb2 = 0, xb3 = 0;
    float sw0 = 0, sw1 = 0, sw2 = 0, sw3 = 0;
    int winL = 0, winM = 0, winP = 0;

    // The window's raw samples are staged with cp.async one multiplet ahead into alternating buffers
    // (4-sample runs: a 4-aligned run never wraps the delay line). Level 0 is read from them.
    Ts *raw0 = (Ts *) (lev + g.raw_off);
    const int raw_ts = g.raw_floats * int(sizeof(float) / sizeof(Ts));
    auto stage = [&](int m) {
        const Ts *row = pfrows + (long) m * a.pf_cap;
        Ts *raw = raw0 + (m & 1) * raw_ts;
        for (int q = lane; q < nq0; q += LW)
            cp_async_bytes<4 * sizeof(Ts)>(raw + 4 * q, row + ((sbm + 4 * q) & mask));
        cp_async_commit();
    };
    stage(0);

    for (int m = 0; m < a.M; m++) {
        // Wait for this multiplet's samples; then stage the next one into the other buffer (every
        // lane is past its reads of that buffer: they came before this loop's previous barriers).
        cp_async_wait0();
        __syncwarp();
        if (m + 1 < a.M)
            stage(m + 1);
        const Ts *rawc = raw0 + (m & 1) * raw_ts;

        const int n = a.m_to_n[m];
        if (n != wsm_n) {
            for (int idx = lane; idx < a.P * NT; idx += LW) {
                const int p = idx / NT, j = idx - p * NT, t = tw0 + j;
                wsm[p * 32 + j] = (t < a.nt_wt) ? wrow[((long) t * a.P + p) * a.N + n] : 0.0f;
            }
            __syncwarp();
            wsm_n = n;
        }
#pragma unroll
        for (int l = 0; l < L; l++) {
            const int S = g.S[l], nsamp = g.nsamp[l];
            const bool U = g.flags[l] & kPfU;
            const bool nextU = (l + 1 < L) && (g.flags[l] & kPfNextU);

            if (l > 0 && !U) {
                // Saturated level (dt = Dcore): B_l[u] = B_{l-1}[rr u] + B_{l-1}[rr u + ss].
                const int rr = g.rr[l], ss = g.ss[l];
                for (int u = lane; u < g.n[l]; u += LW)
                    lev[pf_phys(g, l, u)] = __fadd_rn(lev[pf_phys(g, l - 1, rr * u)], lev[pf_phys(g, l - 1, rr * u + ss)]);
                __syncwarp();
            }
            if (nextU) {
                // Entries of level l+1 before the first output time.
                for (int u = lane; u < g.I[l + 1]; u += LW)
                    lev[pf_phys(g, l + 1, u)] = (l == 0) ? __fadd_rn(to_f(rawc[2 * u]), to_f(rawc[2 * u + 1]))
                                                        : __fadd_rn(lev[pf_phys(g, l, 2 * u)], lev[pf_phys(g, l, 2 * u + 1)]);
            }

            float w0 = 0.0f, w1 = 0.0f, w2 = 0.0f, w3 = 0.0f;
            if (l == 0) w0 = wsm[tl];
            if (full) {
                w1 = wsm[(3 * l + 1) * 32 + tl];
                w2 = wsm[(3 * l + 2) * 32 + tl];
                w3 = wsm[(3 * l + 3) * 32 + tl];
            }

            const int j0 = g.I[l] + lane * nsamp;
            float gmax = -1.0e30f;
            int gp = 0;   // first fine sample (pair start) whose trials reach gmax
            if (g.flags[l] & kPfPairs) {
                // x0..x3 = x[is-3..is]; carried: x2, hx1 = x[is-2]/2, hx2 = x[is-1]/2, Ap = x[is-3]/2 + x[is-2].
                // Level 0 comes from the raw staging buffer (entry i = raw sample i; j0 is a multiple of 4).
                float x2, x1, x0;
                if (l == 0) {
                    float q[4];
                    pf_load4<Ts>(rawc + j0 - 4, q);
                    x0 = q[1]; x1 = q[2]; x2 = q[3];
                } else {
                    x2 = lev[pf_phys(g, l, j0 - 1)];
                    x1 = lev[pf_phys(g, l, j0 - 2)];
                    x0 = lev[pf_phys(g, l, j0 - 3)];
                }
                float2 H = make_float2(__fmul_rn(0.5f, x1), __fmul_rn(0.5f, x2));   // x[is-2]/2, x[is-1]/2
                float Ap = __fadd_rn(__fmul_rn(0.5f, x0), x1);
                const float *xs = lev + ((l > 0) ? pf_phys(g, l, j0) : 0);
                float *ys = lev + (nextU ? pf_phys(g, l + 1, g.I[l + 1] + lane * (nsamp >> 1)) : 0);
                const float2 W0 = make_float2(w0, w0), W1 = make_float2(w1, w1);
                const float2 W2 = make_float2(w2, w2), W3 = make_float2(w3, w3);

                // The trials of fine samples is (xa) and is + 1 (xb).
                auto pair = [&](const float xa, const float xb, const int is) {
                    const float2 X = make_float2(xa, xb);
                    float mx;
                    if (full) {
                        // Fine samples is (xa) and is+1 (xb), in packed pairs (a, b): profiles
                        // y1 = x2+x3, y2 = (x1/2+x2)+x3/2, y3 = ((x0/2+x1)+x2)+x3/2 with the reference's
                        // association; A = x1/2+x2 of each sample, and y3's (x0/2+x1) is the previous A.
                        const float2 Hn = f2mul(make_float2(0.5f, 0.5f), X);
                        const float2 Pr = make_float2(x2, xa);       // x[is-1], x[is]
                        const float2 A = f2add(H, Pr);
                        const float2 V1 = f2mul(W1, f2add(Pr, X));
                        const float2 V2 = f2mul(W2, f2add(A, Hn));
                        const float2 V3 = f2mul(W3, f2add(f2add(make_float2(Ap, A.x), Pr), Hn));
                        if (l == 0) {
                            const float2 V0 = f2mul(W0, X);
                            mx = fmaxf(pf_max3(V0.x, V1.x, V2.x), pf_max3(V3.x, V0.y, V1.y));
                            mx = pf_max3(mx, V2.y, V3.y);
                        } else {
                            mx = fmaxf(pf_max3(V1.x, V2.x, V3.x), pf_max3(V1.y, V2.y, V3.y));
                        }
                        H = Hn; x2 = xb; Ap = A.y;
                    } else {
                        mx = fmaxf(__fmul_rn(w0, xa), __fmul_rn(w0, xb));
                    }
                    if (mx > gmax) { gmax = mx; gp = is; }
                    if (nextU) ys[is >> 1] = __fadd_rn(xa, xb);
                };
                if (l == 0) {
                    // 16-byte loads when runs of 8 stay 16-byte aligned (tpad and Dout multiples of 8)
                    if (DOUT > 0 && nsamp % 8 == 0 && pf_tpad_of(L) % 8 == 0) {
                        for (int is = 0; is < nsamp; is += 8) {
                            float q[8];
                            pf_load8<Ts>(rawc + j0 + is, q);
                            pair(q[0], q[1], is);
                            pair(q[2], q[3], is + 2);
                            pair(q[4], q[5], is + 4);
                            pair(q[6], q[7], is + 6);
                        }
                    } else {
                        for (int is = 0; is < nsamp; is += 4) {
                            float q[4];
                            pf_load4<Ts>(rawc + j0 + is, q);
                            pair(q[0], q[1], is);
                            pair(q[2], q[3], is + 2);
                        }
                    }
                } else {
#pragma unroll 2
                    for (int is = 0; is < nsamp; is += 2) {
                        const float2 X = *(const float2 *) (xs + is);
                        pair(X.x, X.y, is);
                    }
                }
            } else {
                // Levels stored without padding (contiguous across lanes): x[j - k S] = xb[is - k S].
                const float *xb = lev + pf_phys(g, l, j0);
                if (nsamp >= 2) {
                    // Two fine samples at a time (S and nsamp even: 8-byte aligned pairs).
                    for (int is = 0; is < nsamp; is += 2) {
                        const float2 p3 = *(const float2 *) (xb + is), p2 = *(const float2 *) (xb + is - S);
                        const float2 p1 = *(const float2 *) (xb + is - 2 * S), p0 = *(const float2 *) (xb + is - 3 * S);
                        float mx;
                        if (full) {
                            const float ha = __fmul_rn(0.5f, p3.x), hb = __fmul_rn(0.5f, p3.y);
                            const float v1a = __fmul_rn(w1, __fadd_rn(p2.x, p3.x));
                            const float v2a = __fmul_rn(w2, __fadd_rn(__fadd_rn(__fmul_rn(0.5f, p1.x), p2.x), ha));
                            const float v3a = __fmul_rn(w3, __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(0.5f, p0.x), p1.x), p2.x), ha));
                            const float v1b = __fmul_rn(w1, __fadd_rn(p2.y, p3.y));
                            const float v2b = __fmul_rn(w2, __fadd_rn(__fadd_rn(__fmul_rn(0.5f, p1.y), p2.y), hb));
                            const float v3b = __fmul_rn(w3, __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(0.5f, p0.y), p1.y), p2.y), hb));
                            mx = fmaxf(pf_max3(v1a, v2a, v3a), pf_max3(v1b, v2b, v3b));
                            if (l == 0) mx = pf_max3(mx, __fmul_rn(w0, p3.x), __fmul_rn(w0, p3.y));
                        } else {
                            mx = fmaxf(__fmul_rn(w0, p3.x), __fmul_rn(w0, p3.y));
                        }
                        if (mx > gmax) { gmax = mx; gp = is; }
                    }
                } else {
                    const float x3 = xb[0];
                    float v = (l == 0) ? __fmul_rn(w0, x3) : -1.0e30f;
                    if (full) {
                        const float x0 = xb[-3 * S], x1 = xb[-2 * S], x2 = xb[-S];
                        const float hx3 = __fmul_rn(0.5f, x3);
                        const float y1 = __fadd_rn(x2, x3);
                        const float y2 = __fadd_rn(__fadd_rn(__fmul_rn(0.5f, x1), x2), hx3);
                        const float y3 = __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(0.5f, x0), x1), x2), hx3);
                        v = fmaxf(v, pf_max3(__fmul_rn(w1, y1), __fmul_rn(w2, y2), __fmul_rn(w3, y3)));
                    }
                    if (v > gmax) { gmax = v; gp = 0; }
                }
            }
            __syncwarp();

            const int G = l * a.M + m;
            if (gmax > best || (gmax == best && G < winG)) {
                best = gmax;
                winG = G;
                winL = l;
                winM = m;
                winP = gp;
                const int S = g.S[l];
                const int j = g.I[l] + lane * nsamp + gp;
                // level l's entry i (level 0: the raw sample)
                auto X = [&](int i) { return (l == 0) ? to_f(rawc[i]) : lev[pf_phys(g, l, i)]; };
                xa3 = X(j);
                if (full) {
                    xa2 = X(j - S);
                    xa1 = X(j - 2 * S);
                    xa0 = X(j - 3 * S);
                }
                if (gp + 1 < nsamp) {
                    xb3 = X(j + 1);
                    if (full) {
                        xb2 = X(j + 1 - S);
                        xb1 = X(j + 1 - 2 * S);
                        xb0 = X(j + 1 - 3 * S);
                    }
                }
                sw0 = w0; sw1 = w1; sw2 = w2; sw3 = w3;
            }
        }

    }

    // The first trial of the winning pair, in the reference's order (fine time, then profile 0, 3l+1,
    // 3l+2, 3l+3), equal to the maximum gives the output value and token.
    if (winG >= 0) {
        const int l = winL;
        const uint32_t dt = uint32_t(gr.dt[l]);
        const int nsamp = gr.nsamp[l];
#pragma unroll
        for (int k = 0; k < 2; k++) {
            if (k == 1 && winP + 1 >= nsamp) break;
            const float x3 = k ? xb3 : xa3, x2 = k ? xb2 : xa2, x1 = k ? xb1 : xa1, x0 = k ? xb0 : xa0;
            const uint32_t tk0 = (uint32_t(winM) << 16) | (uint32_t(winP + k) * dt);
            if (l == 0) {
                const float v0 = __fmul_rn(sw0, x3);
                if (v0 == best) { outv = v0; tok = tk0; break; }
            }
            if (full) {
                const float hx3 = __fmul_rn(0.5f, x3);
                const float v1 = __fmul_rn(sw1, __fadd_rn(x2, x3));
                const float v2 = __fmul_rn(sw2, __fadd_rn(__fadd_rn(__fmul_rn(0.5f, x1), x2), hx3));
                const float v3 = __fmul_rn(sw3, __fadd_rn(__fadd_rn(__fadd_rn(__fmul_rn(0.5f, x0), x1), x2), hx3));
                if (v1 == best) { outv = v1; tok = tk0 | (uint32_t(3 * l + 1) << 8); break; }
                if (v2 == best) { outv = v2; tok = tk0 | (uint32_t(3 * l + 2) << 8); break; }
                if (v3 == best) { outv = v3; tok = tk0 | (uint32_t(3 * l + 3) << 8); break; }
            }
        }
    }

    if (!active)
        return;
    const long o = ((long) b * a.ndm_out + dm) * a.nt_out + tout;
    ((Ts *) a.out_max)[o] = from_f<Ts>(outv);
    a.out_argmax[o] = tok;
}

// DOUT > 0: compiled for that output time downsampling (with Dcore = min(DOUT, 8) and the plan's tpad
// for L levels); DOUT = 0: any Dout >= 4, geometry read from the launch arguments.
template<typename Ts, int L, int DOUT, bool CTR, int LW = 32>
__global__ void __launch_bounds__(kPfWarps * 32) pf_fast_kernel(PfArgs a, PfGeom gr)
{
    if constexpr (DOUT > 0) {
        constexpr PfGeom gc = pf_geom(DOUT, pf_dcore_of(DOUT), pf_tpad_of(L), L, sizeof(Ts), LW);
        pf_fast_body<Ts, L, DOUT, CTR, LW>(a, gc, gr);
    } else {
        pf_fast_body<Ts, L, 0, CTR, LW>(a, gr, gr);
    }
}


// -------------------------------------------------------------------------------------------------
// Host launchers.


template<typename Ts, int NLEV>
static void launch_grid_lds_t(const GridLdsArgs &a, cudaStream_t s)
{
    constexpr int W0 = ((1 << NLEV) > 8) ? (1 << NLEV) : 8;
    if (a.T % W0) throw std::runtime_error("grid_lds_kernel: chunk length not a multiple of the window");
    const long nwin = a.T / W0;
    long nthr = nwin * (1L << (a.rank - 1)) * a.B;
    // Blocks start at a window 0 (a multiple of nwin threads, about 128), so that every other window's
    // predecessor is computed in the same block.
    const int target = (a.block_target > 0) ? std::min(a.block_target, kGridMaxThreads) : 128;
    int bd = (nwin <= target) ? int(nwin * (target / nwin)) : (nwin <= kGridMaxThreads ? int(nwin) : kGridMaxThreads);
    if (a.q_data) {
        if (a.T % 256) throw std::runtime_error("grid_lds_kernel: int4 input needs a chunk length that is a multiple of 256");
        grid_lds_kernel<Ts, NLEV, true><<<(unsigned) ((nthr + bd - 1) / bd), bd, 0, s>>>(a);
    } else {
        grid_lds_kernel<Ts, NLEV, false><<<(unsigned) ((nthr + bd - 1) / bd), bd, 0, s>>>(a);
    }
    check_launch("grid_lds_kernel");
}

template<typename Ts>
static void launch_grid_lds_d(const GridLdsArgs &a, cudaStream_t s)
{
    switch (a.nlev) {
    case 0: launch_grid_lds_t<Ts, 0>(a, s); break;
    case 1: launch_grid_lds_t<Ts, 1>(a, s); break;
    case 2: launch_grid_lds_t<Ts, 2>(a, s); break;
    case 3: launch_grid_lds_t<Ts, 3>(a, s); break;
    case 4: launch_grid_lds_t<Ts, 4>(a, s); break;
    case 5: launch_grid_lds_t<Ts, 5>(a, s); break;
    case 6: launch_grid_lds_t<Ts, 6>(a, s); break;
    default: throw std::runtime_error("grid_lds_kernel: unsupported number of levels");
    }
}

void launch_grid_lds(const GridLdsArgs &a, int dtype, cudaStream_t s)
{
    if (a.rank < 1) throw std::runtime_error("grid_lds_kernel: tree rank must be >= 1");
    if (dtype == 0) launch_grid_lds_d<float>(a, s);
    else if (dtype == 1) launch_grid_lds_d<__half>(a, s);
    else launch_grid_lds_d<__nv_bfloat16>(a, s);
}

void launch_stage1(const Stage1Args &a, int dtype, int nblocks, int B, cudaStream_t s)
{
    if (a.in_lag0 != 0 || a.in_lag1 != 0) throw std::runtime_error("launch_stage1: input rows must be aligned (no read lag)");
    if (dtype == 0) launch_stage1_halo_f32(a, nblocks, B, s);
    else if (dtype == 1) launch_stage1_halo_f16(a, nblocks, B, s);
    else launch_stage1_halo_bf16(a, nblocks, B, s);
}

static bool stage2_full_band(const Stage2Args &a)
{
    for (int l = 0; l < split_rb(a.rank) && l < 5; l++)
        if (a.sb_count[l] != 0) return false;
    return true;
}

bool stage2_same_kernel(const Stage2Args &x, const Stage2Args &y)
{
    return x.rank == y.rank && stage2_full_band(x) == stage2_full_band(y);
}

void launch_stage2_multi(const Stage2Args *a, const int *nblocks, int n, int dtype, int B, cudaStream_t s)
{
    if (n < 1 || n > kStage2MaxTrees) throw std::runtime_error("launch_stage2_multi: bad tree count " + std::to_string(n));
    Stage2Multi m;
    memset(&m, 0, sizeof(m));
    m.n = n;
    long tot = 0;
    for (int i = 0; i < n; i++) {
        if (!stage2_same_kernel(a[0], a[i])) throw std::runtime_error("launch_stage2_multi: trees need different kernels");
        if (nblocks[i] < 1) throw std::runtime_error("launch_stage2_multi: bad block count");
        m.t[i] = a[i];
        m.blk0[i] = int(tot);
        tot += nblocks[i];
    }
    if (tot > (1L << 30)) throw std::runtime_error("launch_stage2_multi: grid too large");
    m.blk0[n] = int(tot);
    const bool sub = !stage2_full_band(a[0]);
    if (dtype == 0) launch_stage2_halo_f32(m, sub, int(tot), B, s);
    else if (dtype == 1) launch_stage2_halo_f16(m, sub, int(tot), B, s);
    else launch_stage2_halo_bf16(m, sub, int(tot), B, s);
}

void launch_stage2(const Stage2Args &a, int dtype, int nblocks, int B, cudaStream_t s)
{
    launch_stage2_multi(&a, &nblocks, 1, dtype, B, s);
}

int pf_warp_floats(int Dout, int tpad, int Dcore, int L)
{
    int len0 = 32 * Dout + tpad, tot = 0;
    for (int l = 0; l < L; l++) {
        int dt = (Dcore < (1 << l)) ? Dcore : (1 << l);
        tot += (len0 - (1 << l)) / dt + 1;
    }
    return tot;
}


// The fast kernel needs 4-sample runs of the window (Dout >= 4, tpad and s0 multiples of 4).
static bool pf_fast_ok(const PfArgs &a)
{
    const long s0 = a.chunk_ctr ? (long) a.nt_chunk : a.s0;   // with a counter, s0 is a multiple of nt_chunk
    return !a.force_general && a.Dout >= 4 && (a.tpad % 4) == 0 && (s0 % 4) == 0 && (a.pf_cap % 4) == 0 && a.L <= 5 && a.P <= kPfMaxProfiles;
}

template<typename Ts, int L, int DOUT, int LW = 32>
static void launch_pf_fast(const PfArgs &a, const PfGeom &g, int B, cudaStream_t s)
{
    // g: the geometry for LW lanes per coarse DM
    constexpr int G = 32 / LW;
    size_t sm = (size_t) kPfWarps * G * g.warp_floats * sizeof(float);
    dim3 grid((a.nt_out + LW - 1) / LW, (a.ndm_out + kPfWarps * G - 1) / (kPfWarps * G), B);
    if (a.chunk_ctr) {
        set_smem(pf_fast_kernel<Ts, L, DOUT, true, LW>, sm);
        pf_fast_kernel<Ts, L, DOUT, true, LW><<<grid, kPfWarps * 32, sm, s>>>(a, g);
    } else {
        set_smem(pf_fast_kernel<Ts, L, DOUT, false, LW>, sm);
        pf_fast_kernel<Ts, L, DOUT, false, LW><<<grid, kPfWarps * 32, sm, s>>>(a, g);
    }
    check_launch("pf_fast_kernel");
}

template<typename Ts, int L>
static void launch_pf_l(const PfArgs &a, int B, cudaStream_t s)
{
    if (pf_fast_ok(a)) {
        const PfGeom g = pf_geom(a.Dout, a.Dcore, a.tpad, L, (int) sizeof(Ts));
        // Compiled geometries for the usual output downsamplings (pirate's default Dout = 2^pf_rank).
        const bool std_geom = (a.Dcore == pf_dcore_of(a.Dout)) && (a.tpad == pf_tpad_of(L));
        // Trees with 16 or 8 output times per chunk (the most downsampled primary trees) share a warp
        // between 2 or 4 coarse DMs, so that no lane idles (compiled for the benchmark's Dout 16, widths
        // to 32).
        if constexpr (L == 5) {
            if (std_geom && a.Dout == 16 && a.nt_out <= 8) {
                launch_pf_fast<Ts, L, 16, 8>(a, pf_geom(a.Dout, a.Dcore, a.tpad, L, (int) sizeof(Ts), 8), B, s);
                return;
            }
            if (std_geom && a.Dout == 16 && a.nt_out <= 16) {
                launch_pf_fast<Ts, L, 16, 16>(a, pf_geom(a.Dout, a.Dcore, a.tpad, L, (int) sizeof(Ts), 16), B, s);
                return;
            }
        }
        if (std_geom && a.Dout == 16) launch_pf_fast<Ts, L, 16>(a, g, B, s);
        else if (std_geom && a.Dout == 8) launch_pf_fast<Ts, L, 8>(a, g, B, s);
        else if (std_geom && a.Dout == 4) launch_pf_fast<Ts, L, 4>(a, g, B, s);
        else launch_pf_fast<Ts, L, 0>(a, g, B, s);
        return;
    }
    int wf = pf_warp_floats(a.Dout, a.tpad, a.Dcore, a.L);
    size_t sm = (size_t) kPfWarps * wf * sizeof(float);
    set_smem(pf_kernel<Ts, L>, sm);
    dim3 grid((a.nt_out + 31) / 32, (a.ndm_out + kPfWarps - 1) / kPfWarps, B);
    pf_kernel<Ts, L><<<grid, kPfWarps * 32, sm, s>>>(a, wf);
    check_launch("pf_kernel");
}

template<typename Ts>
static void launch_pf_t(const PfArgs &a, int B, cudaStream_t s)
{
    switch (a.L) {
    case 1: launch_pf_l<Ts, 1>(a, B, s); break;
    case 2: launch_pf_l<Ts, 2>(a, B, s); break;
    case 3: launch_pf_l<Ts, 3>(a, B, s); break;
    case 4: launch_pf_l<Ts, 4>(a, B, s); break;
    case 5: launch_pf_l<Ts, 5>(a, B, s); break;
    default: throw std::runtime_error("pf_kernel: unsupported number of boxcar levels");
    }
}

void launch_pf(const PfArgs &a, int dtype, int B, cudaStream_t s)
{
    if (a.Dout > 64 || a.Dout < 1) throw std::runtime_error("pf_kernel: time downsampling must be in [1, 64]");
    if (dtype == 0) launch_pf_t<float>(a, B, s);
    else if (dtype == 1) launch_pf_t<__half>(a, B, s);
    else launch_pf_t<__nv_bfloat16>(a, B, s);
}

}  // namespace pb2
