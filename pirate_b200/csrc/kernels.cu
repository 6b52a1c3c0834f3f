// kernels.cu -- sm_100a kernels of the B200 dedispersion path.
//
//   grid_warp_kernel, grid_lds_kernel  tree gridding + lagged downsampling (replace GpuTreeGriddingKernel,
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
// grid_lds_kernel, for the chunk lengths, level counts and int4 plans that grid_warp_kernel below does not take
// (grid_warp_ok): one thread per (beam, tree-channel pair (2c, 2c+1), window of W0 level-0 samples); consecutive
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
            for (long i = lo + threadIdx.x; i < hi; i += 4L * blockDim.x) {
                float v[4];
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    const long ii = i + (long) u * blockDim.x;
                    v[u] = (ii < hi) ? to_f(x[ii]) : -INFINITY;
                }
#pragma unroll
                for (int u = 0; u < 4; u++) {
                    nan |= (v[u] != v[u]);
                    if (v[u] > p.v) { p.v = v[u]; p.i = int(i + (long) u * blockDim.x); }
                }
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
    // Threads per block: one round of four loads each over a slice of the largest tree (2000 beams of 1024 values: 51 us
    // with 1024 threads, 19 us so).
    long work = 128;
    for (int t = 0; t < a.ntrees; t++) {
        const long n = a.ndm[t] * a.nt[t], vec = dtype == 0 ? 4 : 8;
        work = std::max(work, (n + C - 1) / C / (4 * (n % vec == 0 ? vec : 1)));
    }
    cudaLaunchConfig_t cfg = {};
    cfg.gridDim = dim3((unsigned) nbeams * C);
    cfg.blockDim = dim3((unsigned) std::min(1024L, (work + 31) / 32 * 32));
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
    if (live) {
        grid_run<Ts, W0, Q>(a, b, 2 * c, t0, r0);
        grid_run<Ts, W0, Q>(a, b, 2 * c + 1, t0, r1);
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

// ---------------------------------------------------------------------------------------------
// The same by one warp per (beam, tree-channel pair): it goes through the chunk in steps of 32 windows of W samples, a
// lane owning one window. The sample before a window comes from the lane before, and before a step from the step
// before, so that nothing is exchanged between warps; the outputs leave in contiguous runs, through the warp's own
// shared memory (written by each lane for its window, a level row's samples would be 2-byte stores 4 to 16 bytes
// apart). The two channels of the pair are the halves of packed fp32 operations.
//
// int4 input goes through tables: an input sample is read by about 2.5 pairs at rank 16 from 16384 channels, so
// per step the warp tabulates, for each input row of the pair and 256-sample scale block, the 16 values that a nibble
// can take, rounded to the storage type; a sample is then a nibble extract and a shared-memory lookup.
//
// What bounds it: instruction issue (two thirds of the slots; 770 warp instructions per pair and 512-sample step with
// int4 input and four levels) and the loads' latency at 20 to 32 warps per SM; the launch bounds are the fastest of those
// tried. Against a thread per window (grid_lds_kernel, with 64-bit divisions to find its window, a block barrier and level
// rows stored 2 bytes at a time), per chunk on a B200: 4 beams of rank 16, int4 to fp16, four levels 661 -> 480 us; 1 beam
// of rank 16, fp32, four levels 313 -> 200 us; 2 beams of rank 16, fp16, no level 297 -> 128 us; 16 beams of rank 12, fp16,
// two levels 215 -> 129 us. Staging the rows of 8 pairs in shared memory, each input sample read and dequantized once,
// took 912, 264, 146 and 141 us: the pairs share too few rows to pay for the barriers.

constexpr int kGridWarps = 4;   // warps per block: consecutive pairs, which share input rows
constexpr int kLutRows = 8;     // input rows of a pair served by the tables

// Packed fp32 pairs: each element is rounded to nearest like the scalar operation.
__device__ __forceinline__ unsigned long long f2bits(float2 a)
{
    unsigned long long r;
    asm("mov.b64 %0, {%1, %2};" : "=l"(r) : "f"(a.x), "f"(a.y));
    return r;
}
__device__ __forceinline__ float2 f2from(unsigned long long r)
{
    float2 d;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(d.x), "=f"(d.y) : "l"(r));
    return d;
}
__device__ __forceinline__ float2 f2bfly(float2 a, float2 b)
{
    unsigned long long s, d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(s) : "l"(f2bits(a)), "l"(f2bits(b)));
    asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(s), "l"(f2bits(make_float2(kRsqrt2, kRsqrt2))));
    return f2from(d);
}
__device__ __forceinline__ float2 f2fma(float2 a, float2 b, float2 c)
{
    unsigned long long d;
    asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(d) : "l"(f2bits(a)), "l"(f2bits(b)), "l"(f2bits(c)));
    return f2from(d);
}

__device__ __forceinline__ float2 f2add(float2 a, float2 b)
{
    unsigned long long d;
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(f2bits(a)), "l"(f2bits(b)));
    return f2from(d);
}

// W samples of one input row as they lie in memory; zeros when !ok.
template<typename Ts, int W>
struct GridRow
{
    uint4 q[W * sizeof(Ts) / 16];
    __device__ __forceinline__ void load(const Ts *p, bool ok)
    {
#pragma unroll
        for (int v = 0; v < int(W * sizeof(Ts) / 16); v++) q[v] = ok ? ((const uint4 *) p)[v] : make_uint4(0, 0, 0, 0);
    }
    __device__ __forceinline__ float get(int i) const
    {
        constexpr int PER = 16 / sizeof(Ts);
        const uint4 &u = q[i / PER];
        const int j = i % PER * int(sizeof(Ts)) / 4;
        const uint32_t v = j == 0 ? u.x : j == 1 ? u.y : j == 2 ? u.z : u.w;
        if constexpr (sizeof(Ts) == 4) return __uint_as_float(v);
        else if constexpr (std::is_same<Ts, __half>::value) return __half2float(__ushort_as_half((unsigned short) (v >> (i & 1) * 16)));
        else return __uint_as_float((i & 1) ? (v & 0xffff0000u) : (v << 16));
    }
};
// Two samples as one word of a 16-bit type.
template<typename Ts>
__device__ __forceinline__ uint32_t pack2(float x, float y)
{
    if constexpr (std::is_same<Ts, __half>::value) {
        const __half2 h = __floats2half2_rn(x, y);
        return *(const uint32_t *) &h;
    } else {
        const __nv_bfloat162 h = __floats2bfloat162_rn(x, y);
        return *(const uint32_t *) &h;
    }
}

// N samples (a power of two) to p, in stores of up to 16 bytes.
template<typename Ts, int N>
__device__ __forceinline__ void store_vec(Ts *p, const float (&o)[N])
{
    if constexpr (sizeof(Ts) == 4) {
        if constexpr (N >= 4) {
#pragma unroll
            for (int i = 0; i < N; i += 4) *(float4 *) (p + i) = make_float4(o[i], o[i + 1], o[i + 2], o[i + 3]);
        } else if constexpr (N == 2) {
            *(float2 *) p = make_float2(o[0], o[1]);
        } else {
            *p = o[0];
        }
    } else {
        if constexpr (N >= 8) {
#pragma unroll
            for (int i = 0; i < N; i += 8)
                *(uint4 *) (p + i) = make_uint4(pack2<Ts>(o[i], o[i + 1]), pack2<Ts>(o[i + 2], o[i + 3]), pack2<Ts>(o[i + 4], o[i + 5]),
                                                pack2<Ts>(o[i + 6], o[i + 7]));
        } else if constexpr (N == 4) {
            *(uint2 *) p = make_uint2(pack2<Ts>(o[0], o[1]), pack2<Ts>(o[2], o[3]));
        } else if constexpr (N == 2) {
            *(uint32_t *) p = pack2<Ts>(o[0], o[1]);
        } else {
            *p = from_f<Ts>(o[0]);
        }
    }
}

template<typename Ts, int NLEV, int W, bool Q>
struct GridWarp
{
    static constexpr int STEP = 32 * W;
    static constexpr int NBLK = STEP / 256;                                   // scale blocks per step
    static constexpr int LUT = Q ? kLutRows * NBLK * 16 * int(sizeof(float)) : 0;
    static constexpr int OUT = STEP * int(sizeof(Ts));
    static constexpr int BYTES = LUT > OUT ? LUT : OUT;                       // shared memory: the tables, then the outputs
    // First sample of level p's row in the output buffer.
    __host__ __device__ static constexpr int off(int p) { return STEP - (STEP >> (p - 1)); }
};

// The warp's 32 windows of W samples to p and on, through buf: 16-byte chunk c lies at c ^ (c / 8 mod CH), which leaves
// neither side bank conflicts.
template<typename Ts, int W>
__device__ __forceinline__ void store_warp(Ts *p, const float (&o)[W], unsigned char *buf, int lane)
{
    constexpr int PER = 16 / sizeof(Ts), CH = W / PER;
    if constexpr (CH == 1) {
        store_vec<Ts, W>(p + lane * W, o);
    } else {
        auto at = [&](int c) { return (uint4 *) buf + (c ^ ((c >> 3) & (CH - 1))); };
#pragma unroll
        for (int v = 0; v < CH; v++) {
            float x[PER];
#pragma unroll
            for (int i = 0; i < PER; i++) x[i] = o[v * PER + i];
            store_vec<Ts, PER>((Ts *) at(lane * CH + v), x);
        }
        __syncwarp();
#pragma unroll
        for (int v = 0; v < CH; v++) ((uint4 *) p)[v * 32 + lane] = *at(v * 32 + lane);
        __syncwarp();
    }
}

// The warp's N samples lev[0..N) (N a multiple of 16) to delay-line positions pos and on. 16-bit types move as words,
// across the halves of two words where the first position is odd.
template<typename Ts, int N>
__device__ __forceinline__ void store_line(Ts *ring, int pos, int mask, const Ts *lev, int lane)
{
    if constexpr (sizeof(Ts) == 4) {
#pragma unroll
        for (int i0 = 0; i0 < N; i0 += 32) {
            const int i = i0 + lane;
            if (N % 32 == 0 || i < N) ring[(pos + i) & mask] = lev[i];
        }
    } else {
        const uint32_t *w = (const uint32_t *) lev + lane;
        uint32_t *o = (uint32_t *) ring;
        const int p2 = (pos >> 1) + lane, m2 = mask >> 1;
        if (pos & 1) {
#pragma unroll
            for (int j0 = 0; j0 < N / 2; j0 += 32)
                if ((j0 > 0 || lane > 0) && (j0 + 32 <= N / 2 || j0 + lane < N / 2)) o[(p2 + j0) & m2] = __byte_perm(w[j0 - 1], w[j0], 0x5432);
            if (lane < 2) ring[(pos + lane * (N - 1)) & mask] = lev[lane * (N - 1)];
        } else {
#pragma unroll
            for (int j0 = 0; j0 < N / 2; j0 += 32)
                if (j0 + 32 <= N / 2 || j0 + lane < N / 2) o[(p2 + j0) & m2] = w[j0];
        }
    }
}

// Levels p .. NLEV of a window, in place as in grid_lds_kernel, into the warp's rows. carry: the even channel's last
// sample of every level before the step.
template<typename Ts, int NLEV, int p, int W>
__device__ __forceinline__ void warp_levels(float2 (&r)[W], float (&carry)[NLEV], Ts *lev, int lane)
{
    constexpr int len = W >> p;
    float o[len];
#pragma unroll
    for (int u = 0; u < len; u++) r[u] = f2bfly(r[2 * u], r[2 * u + 1]);
    const float up = __shfl_up_sync(0xffffffffu, r[len - 1].x, 1);
    o[0] = bfly(lane == 0 ? carry[p - 1] : up, r[0].y);
    carry[p - 1] = __shfl_sync(0xffffffffu, r[len - 1].x, 31);
#pragma unroll
    for (int u = 1; u < len; u++) o[u] = bfly(r[u - 1].x, r[u].y);
    store_vec<Ts, len>(lev + GridWarp<Ts, NLEV, W, false>::off(p) + lane * len, o);
    if constexpr (p < NLEV) warp_levels<Ts, NLEV, p + 1, W>(r, carry, lev, lane);
}

template<typename Ts, int NLEV, int p, int W>
__device__ __forceinline__ void warp_lines(const GridLdsArgs &a, long row, unsigned u, unsigned lag, const Ts *lev, int lane)
{
    // row: the pair's row of the delay lines; u: the step's first level-0 sample (its low bits)
    using G = GridWarp<Ts, NLEV, W, false>;
    const int mask = int(a.cap_mask[p - 1]);
    store_line<Ts, (G::STEP >> p)>((Ts *) a.ring[p - 1] + row * (mask + 1), int((u >> p) + lag) & mask, mask, lev + G::off(p), lane);
    if constexpr (p < NLEV) warp_lines<Ts, NLEV, p + 1, W>(a, row, u, lag, lev, lane);
}

// Sample k8 of a nibble word, from the table at shared address L (a multiple of 64).
__device__ __forceinline__ float lut_at(uint32_t L, uint32_t q, int k8)
{
    float v;
    asm volatile("ld.shared.f32 %0, [%1];" : "=f"(v) : "r"(L | ((k8 ? q >> (4 * k8 - 2) : q << 2) & 0x3cu)));
    return v;
}

// The nibble words of W samples at p.
template<int W>
__device__ __forceinline__ void lut_words(const unsigned char *p, uint32_t (&q)[W / 8])
{
    if constexpr (W == 16) {
        const uint2 w = *(const uint2 *) p;
        q[0] = w.x;
        q[1] = w.y;
    } else {
        q[0] = *(const uint32_t *) p;
    }
}

// WIDE: plans with at least as many input channels as tree channels (not for int4).
template<typename Ts, int NLEV, int W, bool Q, bool WIDE>
__global__ void __launch_bounds__(32 * kGridWarps, W == 16 ? (Q ? 6 : 5) : 8) grid_warp_kernel(GridLdsArgs a)
{
    using G = GridWarp<Ts, NLEV, W, Q>;
    constexpr int STEP = G::STEP;
    __shared__ __align__(128) unsigned char grid_sm[kGridWarps * G::BYTES];
    const int lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    unsigned char *wsm = grid_sm + warp * G::BYTES;
    const int nhalf = 1 << (a.rank - 1);
    const int c = blockIdx.x * kGridWarps + warp, b = blockIdx.y, bt = a.beam0 + b;
    if (c >= nhalf) return;   // whole warps; nothing below waits for another warp
    const long ichunk = a.chunk_ctr ? *a.chunk_ctr : a.ichunk;
    const int parity = int(ichunk & 1);
    // This warp's steps: a share of the chunk's where pairs alone are too few for the GPU.
    const int nsteps = a.T / STEP;
    const int s0 = nsteps * int(blockIdx.z) / int(gridDim.z), s1 = nsteps * (int(blockIdx.z) + 1) / int(gridDim.z);

    const int fa = a.chan_f0[2 * c], ca = a.chan_cnt[2 * c], fb = a.chan_f0[2 * c + 1], cb = a.chan_cnt[2 * c + 1];
    const float *wa = a.chan_w + a.chan_woff[2 * c], *wb = a.chan_w + a.chan_woff[2 * c + 1];
    const float2 w0 = make_float2(ca > 0 ? wa[0] : 0.0f, cb > 0 ? wb[0] : 0.0f);
    Ts *tree = (Ts *) a.tree0 + ((long) b * (2 * nhalf) + 2 * c) * a.T;

    float carry[NLEV > 0 ? NLEV : 1];
    const unsigned u0 = unsigned(ichunk * a.T);   // low bits of the chunk's first sample: delay lines have fewer than 2^27 slots
    const unsigned lag = (1u << a.lag_rank) - 1 - (c & ((1u << a.lag_rank) - 1));
    if constexpr (NLEV > 0) {
        if (s0 == 0) {
#pragma unroll
            for (int p = 1; p <= NLEV; p++)
                carry[p - 1] = a.state[(((long) parity * a.total_beams + bt) * a.nlev + (p - 1)) * nhalf + c];
        } else {
            // the even channel's 2^NLEV samples before, one per lane
            constexpr int WE = 1 << NLEV;
            float e[1];
            grid_run<Ts, 1, Q>(a, b, 2 * c, (long) s0 * STEP - WE + (lane & (WE - 1)), e);
#pragma unroll
            for (int p = 1; p <= NLEV; p++) {
                e[0] = bfly(e[0], __shfl_xor_sync(0xffffffffu, e[0], 1 << (p - 1)));
                carry[p - 1] = __shfl_sync(0xffffffffu, e[0], WE - 1);
            }
        }
    }

    // int4: the pair's input rows from rlo on, if they fit the tables, and the step's words of the first ones.
    const int rlo = min(ca ? fa : fb, cb ? fb : fa), rows = max(fa + ca, fb + cb) - rlo;
    const bool use_lut = Q && rows <= kLutRows;
    const unsigned char *qa = nullptr, *qb = nullptr;
    const __half2 *so = nullptr;
    uint32_t la = 0, lb = 0, va[W / 8], vb[W / 8];
    float fv = 0.0f;
    if constexpr (Q) {
        const unsigned char *q = (const unsigned char *) a.q_data + (long) b * a.F * (a.T >> 1) + (s0 * STEP + lane * W) / 2;
        qa = q + (long) (ca ? fa : rlo) * (a.T >> 1);
        qb = q + (long) (cb ? fb : rlo) * (a.T >> 1);
        so = (const __half2 *) a.q_scoff + ((long) b * a.F + rlo) * (a.T >> 8) + ((s0 * STEP) >> 8) + (G::NBLK == 2 ? lane >> 4 : 0);
        const uint32_t L = (uint32_t) __cvta_generic_to_shared(wsm) + (G::NBLK == 2 ? (lane >> 4) * 64 : 0);
        la = L + (ca ? fa - rlo : 0) * G::NBLK * 64;
        lb = L + (cb ? fb - rlo : 0) * G::NBLK * 64;
        fv = float(((lane & 15) ^ 8) - 8);   // the nibble this lane tabulates
        if (use_lut) {
            lut_words<W>(qa, va);
            lut_words<W>(qb, vb);
        }
    }

    for (int s = s0; s < s1; s++) {
        const int t0 = s * STEP + lane * W;
        float2 r[W];   // the channels' samples: even (x) and odd (y)
        if (use_lut) {
#pragma unroll 1
            for (int k = 0; k < rows; k += 2) {
                __half2 p[2];
#pragma unroll
                for (int g = 0; g < 2; g++) p[g] = so[(long) min(k + g, rows - 1) * (a.T >> 8)];
#pragma unroll
                for (int g = 0; g < 2; g++) {
                    const float2 sc = __half22float2(p[g]);
                    const float x = (lane & 15) == 8 ? 0.0f : to_f(from_f<Ts>(__fadd_rn(__fmul_rn(sc.x, fv), sc.y)));
                    if (G::NBLK == 2 || lane < 16) ((float *) wsm)[min(k + g, rows - 1) * G::NBLK * 16 + lane] = x;
                }
            }
            so += G::NBLK;
            __syncwarp();
            // The first row's products are added to zero by one fused multiply-add, which rounds like the product.
#pragma unroll
            for (int i = 0; i < W; i++)
                r[i] = f2fma(w0, make_float2(lut_at(la, va[i / 8], i & 7), lut_at(lb, vb[i / 8], i & 7)), make_float2(0.0f, 0.0f));
            if (ca == 0 || cb == 0)   // a channel without input is zero, whatever the tables hold
#pragma unroll
                for (int i = 0; i < W; i++) r[i] = make_float2(ca ? r[i].x : 0.0f, cb ? r[i].y : 0.0f);
#pragma unroll 1
            for (int k = 1; k < max(ca, cb); k++) {
                if (k < ca) lut_words<W>(qa + (long) k * (a.T >> 1), va);
                if (k < cb) lut_words<W>(qb + (long) k * (a.T >> 1), vb);
                if (k < ca) {
                    const float wk = wa[k];
#pragma unroll
                    for (int i = 0; i < W; i++) r[i].x = __fadd_rn(r[i].x, __fmul_rn(wk, lut_at(la + k * G::NBLK * 64, va[i / 8], i & 7)));
                }
                if (k < cb) {
                    const float wk = wb[k];
#pragma unroll
                    for (int i = 0; i < W; i++) r[i].y = __fadd_rn(r[i].y, __fmul_rn(wk, lut_at(lb + k * G::NBLK * 64, vb[i / 8], i & 7)));
                }
            }
            qa += STEP / 2;
            qb += STEP / 2;
            if (s + 1 < s1) {
                lut_words<W>(qa, va);
                lut_words<W>(qb, vb);
            }
            __syncwarp();   // the tables' memory is the outputs' from here on
        } else if constexpr (Q) {
            float x[W];
            grid_run<Ts, W, Q>(a, b, 2 * c, t0, x);
#pragma unroll
            for (int i = 0; i < W; i++) r[i].x = x[i];
            grid_run<Ts, W, Q>(a, b, 2 * c + 1, t0, x);
#pragma unroll
            for (int i = 0; i < W; i++) r[i].y = x[i];
        } else if constexpr (WIDE) {
            // Both channels' rows together, in pairs where registers allow, so that their loads are in flight together; a
            // channel past its last row adds 0 * 0.
            constexpr int GR = W * sizeof(Ts) <= 16 ? 2 : 1;
            const Ts *pa = (const Ts *) a.in + ((long) b * a.F + fa) * a.T + t0, *pb = pa + (long) (fb - fa) * a.T;
#pragma unroll
            for (int i = 0; i < W; i++) r[i] = make_float2(0.0f, 0.0f);
#pragma unroll 1
            for (int k = 0; k < max(ca, cb); k += GR) {
                GridRow<Ts, W> x[GR], y[GR];
                float2 w[GR];
#pragma unroll
                for (int g = 0; g < GR; g++) {
                    const bool oka = k + g < ca, okb = k + g < cb;
                    w[g] = make_float2(oka ? wa[k + g] : 0.0f, okb ? wb[k + g] : 0.0f);
                    x[g].load(pa, oka);
                    y[g].load(pb, okb);
                    pa += a.T;
                    pb += a.T;
                }
                // Scalar products: a packed product and the packed sum that takes it came out as one fused operation.
#pragma unroll
                for (int g = 0; g < GR; g++)
#pragma unroll
                    for (int i = 0; i < W; i++) r[i] = f2add(r[i], make_float2(__fmul_rn(w[g].x, x[g].get(i)), __fmul_rn(w[g].y, y[g].get(i))));
            }
        } else {
            const Ts *in = (const Ts *) a.in + (long) b * a.F * a.T + t0;
            float x[W], y[W];
#pragma unroll
            for (int i = 0; i < W; i++) x[i] = y[i] = 0.0f;
            if (ca > 0) load_run<Ts, W>(in + (long) fa * a.T, x);
            if (cb > 0) load_run<Ts, W>(in + (long) fb * a.T, y);
#pragma unroll
            for (int i = 0; i < W; i++) r[i] = f2fma(w0, make_float2(x[i], y[i]), make_float2(0.0f, 0.0f));
#pragma unroll 1
            for (int k = 1; k < ca; k++) {
                load_run<Ts, W>(in + (long) (fa + k) * a.T, x);
                const float wk = wa[k];
#pragma unroll
                for (int i = 0; i < W; i++) r[i].x = __fadd_rn(r[i].x, __fmul_rn(wk, x[i]));
            }
#pragma unroll 1
            for (int k = 1; k < cb; k++) {
                load_run<Ts, W>(in + (long) (fb + k) * a.T, y);
                const float wk = wb[k];
#pragma unroll
                for (int i = 0; i < W; i++) r[i].y = __fadd_rn(r[i].y, __fmul_rn(wk, y[i]));
            }
        }
        float x[W];
#pragma unroll
        for (int i = 0; i < W; i++) x[i] = r[i].x;
        store_warp<Ts, W>(tree + s * STEP, x, wsm, lane);
#pragma unroll
        for (int i = 0; i < W; i++) x[i] = r[i].y;
        store_warp<Ts, W>(tree + a.T + s * STEP, x, wsm, lane);
        if constexpr (NLEV > 0) {
            warp_levels<Ts, NLEV, 1, W>(r, carry, (Ts *) wsm, lane);
            __syncwarp();
            warp_lines<Ts, NLEV, 1, W>(a, (long) bt * nhalf + c, u0 + unsigned(s * STEP), lag, (const Ts *) wsm, lane);
            __syncwarp();
        }
    }
    if (NLEV > 0 && lane == 0 && s1 == nsteps) {
#pragma unroll
        for (int p = 1; p <= NLEV; p++)
            a.state[(((long) (1 - parity) * a.total_beams + bt) * a.nlev + (p - 1)) * nhalf + c] = carry[p - 1];
    }
}

// -------------------------------------------------------------------------------------------------
// Peak finding. One warp per (beam, coarse dm, 32 consecutive output times). For each multiplet m
// the warp stages the input window in shared memory and builds the boxcar levels with the reference's
// recursion  B_{l+1}[u] = B_l[r u] + B_l[r u + s]  (so every boxcar sum has the reference's rounding);
// each lane then scans the trials of its output time. The running maximum breaks ties by the
// reference's scan order (level, multiplet, fine time, profile), reproducing its out_argmax tokens.

constexpr int kPfWarps = 4;

// Number of entries of boxcar level l in a window of len0 samples (level 0 = samples).
__device__ __forceinline__ int pf_nlev(int len0, int l, int dt) { return (len0 - (1 << l)) / dt + 1; }

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
// Host launchers.

template<typename Ts, int NLEV, int W, bool Q>
static void launch_grid_warp(const GridLdsArgs &a, cudaStream_t s)
{
    const int nblk = ((1 << (a.rank - 1)) + kGridWarps - 1) / kGridWarps, nsteps = a.T / (32 * W);
    // Few pairs: split the chunk over up to 8 blocks per SM, or 32 and 64 where a tree channel sums 1 and 4 input
    // channels and more: those of the low end of the band sum three times the average and are the longest chains.
    // 8 beams of rank 10, fp16, 3 trees, 1 input channel per tree channel 33 -> 29 us, 4 115 -> 58, 16 407 -> 152, the
    // rows' loads of WIDE included.
    const int per_sm = a.F >> a.rank >= 4 ? 64 : a.F >> a.rank >= 1 ? 32 : 8;
    const int nz = std::max(1, std::min(nsteps, per_sm * 148 / std::max(1, nblk * a.B)));
    const dim3 grid(nblk, a.B, nz);
    if constexpr (!Q) {
        if (a.F >> a.rank >= 1) {
            grid_warp_kernel<Ts, NLEV, W, Q, true><<<grid, 32 * kGridWarps, 0, s>>>(a);
            check_launch("grid_warp_kernel");
            return;
        }
    }
    grid_warp_kernel<Ts, NLEV, W, Q, false><<<grid, 32 * kGridWarps, 0, s>>>(a);
    check_launch("grid_warp_kernel");
}

template<typename Ts, int NLEV>
static void launch_grid_lds_t(const GridLdsArgs &a, cudaStream_t s)
{
    if (a.q_data && a.T % 256) throw std::runtime_error("grid_lds_kernel: int4 input needs a chunk length that is a multiple of 256");
    if (grid_warp_ok(a.T, NLEV, a.F, a.rank, a.q_data != nullptr)) {
        // A warp per pair for whole steps, faster than a thread per window (1 beam of rank 10 11 -> 10 us, of rank 8 the
        // same; larger ones above grid_warp_kernel), but for int4 input of many channels (see grid_warp_ok). 16-sample windows where the levels need
        // them, and for int4 input, whose tables then have two scale blocks per step for the warp to fill.
        if constexpr (NLEV == 4) {
            if (a.q_data) launch_grid_warp<Ts, NLEV, 16, true>(a, s);
            else launch_grid_warp<Ts, NLEV, 16, false>(a, s);
        } else if constexpr (NLEV < 4) {
            if (!a.q_data) launch_grid_warp<Ts, NLEV, 8, false>(a, s);
            else if (a.T % 512 == 0) launch_grid_warp<Ts, NLEV, 16, true>(a, s);
            else launch_grid_warp<Ts, NLEV, 8, true>(a, s);
        }
        return;
    }
    constexpr int W0 = ((1 << NLEV) > 8) ? (1 << NLEV) : 8;
    if (a.T % W0) throw std::runtime_error("grid_lds_kernel: chunk length not a multiple of the window");
    const long nwin = a.T / W0;
    long nthr = nwin * (1L << (a.rank - 1)) * a.B;
    // Blocks start at a window 0 (a multiple of nwin threads, about 128), so that every other window's
    // predecessor is computed in the same block.
    const int target = (a.block_target > 0) ? std::min(a.block_target, kGridMaxThreads) : 128;
    int bd = (nwin <= target) ? int(nwin * (target / nwin)) : (nwin <= kGridMaxThreads ? int(nwin) : kGridMaxThreads);
    if (a.q_data) {
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

template<typename Ts, int L>
static void launch_pf_l(const PfArgs &a, int B, cudaStream_t s)
{
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
    // The register kernel wherever its geometry applies, that is for every plan with a time downsampling of 2 to 64
    // (measured at 2 to 16: 1 beam of rank 10 15 -> 11 us, 4 beams of rank 16 1434 -> 957 us); the general one for a
    // time downsampling of 1.
    if (pf_reg_ok(a)) {
        if (dtype == 0) launch_pf_reg_f32(a, B, s);
        else if (dtype == 1) launch_pf_reg_f16(a, B, s);
        else launch_pf_reg_bf16(a, B, s);
        return;
    }
    if (dtype == 0) launch_pf_t<float>(a, B, s);
    else if (dtype == 1) launch_pf_t<__half>(a, B, s);
    else launch_pf_t<__nv_bfloat16>(a, B, s);
}

}  // namespace pb2
