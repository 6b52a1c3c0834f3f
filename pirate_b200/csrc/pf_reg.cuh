// pf_reg.cuh -- peak finding in registers.
//
// One warp per (beam, 32 output times) of one coarse dm, or of 2 or 4 coarse dms where a chunk has at most 16 or 8
// output times; a lane owns one output time, i.e. DOUT consecutive samples of every multiplet row. Per multiplet
// the window (the lanes' samples and the tpad before them) is staged in shared memory with cp.async, one to
// three multiplets ahead; a lane reads its own DOUT samples and keeps every boxcar level's entries of them in registers. The
// entries that a profile reaches back to belong to the lanes before and come by shuffle: the lane that holds the
// wanted entry offers it, and the entries before the warp's first output time ("halo") are computed by the last
// lanes of the warp, which offer them in place of their own, since nobody reads those at that distance.
//
// The maximum over a group (level, multiplet) of weight * profile is found without multiplying every trial: with a
// finite weight > 0, rounding is monotone, so the largest product is the product of the largest profile value,
// exactly. A warp with any other weight multiplies every trial. Either way only the maximum per level and the first
// multiplet reaching it are kept; at the end each lane scans its winning group's trials once more, from the row in
// global memory, for the first one (in fine time, then profile order) equal to the maximum: its value and token are
// the outputs. This reproduces ReferencePeakFindingKernel::apply's sequential strict-'>' scan
// (src_lib/PeakFindingKernel.cu:339-420): ties, NaN (never selected) and the sign of zero.
//
// What bounds it: instruction issue (83% of the slots; the rows are read from memory once). A kernel that kept the boxcar
// levels as arrays in shared memory took 47 warp instructions per 32 samples; this one takes 34. Against it, per chunk
// on a B200 (fp16, 112 trials per output): 4 beams of rank 16 with 5 trees 1434 -> 957 us, 16 beams of rank 12
// 477 -> 355 us; 1 beam of rank 16 in fp32 472 -> 338 us. Registers are held to 5 blocks of 4 warps per SM up to
// DOUT = 16, 3 and 2 beyond. The last scan reads its window into registers with vector loads: sample by sample from
// global memory it made the kernel slower than the one it replaces.

#pragma once

#include "kernels.cuh"
#include "devutil.cuh"

#include <type_traits>

namespace pb2 {

constexpr int kPfRegWarps = 4;

template<typename Ts, int L, int DOUT>
struct PfReg
{
    static constexpr int DC = DOUT < 8 ? DOUT : 8;                        // time step of the longest boxcars (Dcore)
    static constexpr int TP = (2 << L) > 4 ? (2 << L) : 4;                // samples before an output time (tpad)
    static constexpr int BB = DOUT * int(sizeof(Ts));                     // bytes per lane and multiplet
    static constexpr int U = BB < 16 ? 16 / BB : 1;                       // lanes per 16-byte chunk
    static constexpr int HL = ((TP + DOUT - 1) / DOUT + U - 1) / U * U;   // halo lanes
    static constexpr int CPL = BB >= 16 ? BB / 16 : 1;                    // chunks per lane
    // Staged multiplets: 3 ahead where a few blocks wait for their loads (4 rank-11 beams, bf16, in two batches: 210 ->
    // 180 us; 16 rank-12 beams 362 -> 355 us), 1 ahead for 64 bytes and more a lane (fp32, DOUT 16: 338 us, 346 with 3).
    static constexpr int NBUF = BB <= 32 ? 4 : 2;
    static constexpr int LWMIN = HL <= 8 ? 8 : HL <= 16 ? 16 : 32;        // fewest lanes per coarse dm
    static_assert(HL <= 32, "halo lanes");
    __host__ __device__ static constexpr int dt(int l) { return (1 << l) < DC ? (1 << l) : DC; }
    __host__ __device__ static constexpr int ns(int l) { return DOUT / dt(l); }
    __host__ __device__ static constexpr int S(int l) { return (1 << l) / dt(l); }
    // Chunk c of a window lies at c ^ swz: the 8 lanes of a 16-byte shared load then touch all banks.
    __host__ __device__ static constexpr int swz(int c) { return c ^ ((c >> 3) & (CPL >= 4 ? 3 : CPL - 1)); }
};

// max(a, b, c) ignoring NaN inputs (sm_100 three-input max).
__device__ __forceinline__ float pfr_max3(float a, float b, float c)
{
    float d;
    asm("max.f32 %0, %1, %2, %3;" : "=f"(d) : "f"(a), "f"(b), "f"(c));
    return d;
}

// DOUT samples of block 'blk' of a staged window.
template<typename Ts, int L, int DOUT>
__device__ __forceinline__ void pfr_load(const unsigned char *win, int blk, float *x)
{
    using R = PfReg<Ts, L, DOUT>;
    if constexpr (R::BB >= 16) {
        constexpr int PER = 16 / sizeof(Ts);
#pragma unroll
        for (int c = 0; c < R::CPL; c++) {
            const uint4 q = *(const uint4 *) (win + 16 * R::swz(blk * R::CPL + c));
            const uint32_t w[4] = {q.x, q.y, q.z, q.w};
#pragma unroll
            for (int i = 0; i < 4; i++) {
                if constexpr (sizeof(Ts) == 4) {
                    x[c * PER + i] = __uint_as_float(w[i]);
                } else {
                    float2 f;
                    if constexpr (std::is_same<Ts, __half>::value) f = __half22float2(*(const __half2 *) &w[i]);
                    else f = make_float2(__uint_as_float(w[i] << 16), __uint_as_float(w[i] & 0xffff0000u));
                    x[c * PER + 2 * i] = f.x;
                    x[c * PER + 2 * i + 1] = f.y;
                }
            }
        }
    } else {
        const Ts *p = (const Ts *) (win + blk * R::BB);
#pragma unroll
        for (int i = 0; i < DOUT; i++) x[i] = to_f(p[i]);
    }
}

// The window of one output time, its DOUT samples and the blocks before them, as raw words of one row: sample i
// (negative: before the output time) by get(i), i a compile-time constant once unrolled.
template<typename Ts, int L, int DOUT>
struct PfWindow
{
    using R = PfReg<Ts, L, DOUT>;
    static constexpr int NB = (R::TP + DOUT - 1) / DOUT + 1;   // blocks
    static constexpr int WPB = R::BB / 4;                      // words per block
    uint32_t w[NB * WPB];
    __device__ __forceinline__ void load(const Ts *row, int t0, int mask)
    {
#pragma unroll
        for (int k = 0; k < NB; k++) {
            const Ts *p = row + ((t0 + (k - (NB - 1)) * DOUT) & mask);
            if constexpr (R::BB >= 16) {
#pragma unroll
                for (int c = 0; c < R::CPL; c++) {
                    const uint4 q = ((const uint4 *) p)[c];
                    w[k * WPB + 4 * c] = q.x;
                    w[k * WPB + 4 * c + 1] = q.y;
                    w[k * WPB + 4 * c + 2] = q.z;
                    w[k * WPB + 4 * c + 3] = q.w;
                }
            } else {
#pragma unroll
                for (int c = 0; c < WPB; c++) w[k * WPB + c] = ((const uint32_t *) p)[c];
            }
        }
    }
    __device__ __forceinline__ float get(int i) const
    {
        const int j = i + (NB - 1) * DOUT;
        if constexpr (sizeof(Ts) == 4) {
            return __uint_as_float(w[j]);
        } else {
            const uint32_t v = w[j >> 1];
            if constexpr (std::is_same<Ts, __half>::value) {
                const __half2 h = *(const __half2 *) &v;
                return (j & 1) ? __high2float(h) : __low2float(h);
            } else {
                return __uint_as_float((j & 1) ? (v & 0xffff0000u) : (v << 16));
            }
        }
    }
    // o[i] = entry U0 + i of level l (entry u ends with sample (u + 1) dt - 1), in the boxcar recursion's order.
    template<int l, int U0, int N>
    __device__ __forceinline__ void entries(float (&o)[N]) const
    {
        if constexpr (l == 0) {
#pragma unroll
            for (int i = 0; i < N; i++) o[i] = get(U0 + i);
        } else if constexpr ((1 << l) <= R::DC) {
            float t[2 * N];
            entries<l - 1, 2 * U0, 2 * N>(t);
#pragma unroll
            for (int i = 0; i < N; i++) o[i] = __fadd_rn(t[2 * i], t[2 * i + 1]);
        } else {
            constexpr int S1 = R::S(l - 1);
            float t[N + S1];
            entries<l - 1, U0 - S1, N + S1>(t);
#pragma unroll
            for (int i = 0; i < N; i++) o[i] = __fadd_rn(t[i], t[i + S1]);
        }
    }
};

// The three profiles that reach back 1, 2 and 3 entries: y1 = x2 + x3, y2 = (x1/2 + x2) + x3/2,
// y3 = ((x0/2 + x1) + x2) + x3/2, with the reference's association. Halving is exact, so a fused multiply-add by 1/2
// rounds like the reference's product and sum (but for subnormal samples, whose halves it does not round).
__device__ __forceinline__ float pfr_half_add(float x, float y) { return __fmaf_rn(0.5f, x, y); }   // x/2 + y

// The first trial of level l equal to 'best' (scanned from the last one back).
template<typename Ts, int L, int DOUT, int l>
__device__ __forceinline__ void pfr_rescan(const PfWindow<Ts, L, DOUT> &win, float w0, float w1, float w2, float w3, bool full, float best,
                                           float &val, uint32_t &tok)
{
    using R = PfReg<Ts, L, DOUT>;
    constexpr int dt = R::dt(l), ns = R::ns(l), S = R::S(l);
    float X[3 * S + ns];
    win.template entries<l, -3 * S, 3 * S + ns>(X);
    auto take = [&](float v, uint32_t t) {
        if (v == best) { val = v; tok = t; }
    };
#pragma unroll
    for (int is = ns - 1; is >= 0; is--) {
        const float *x = X + 3 * S + is;
        const uint32_t t = uint32_t(is * dt);
        const float x3 = x[0];
        if (full) {
            const float x2 = x[-S], x1 = x[-2 * S], x0 = x[-3 * S];
            take(__fmul_rn(w3, pfr_half_add(x3, __fadd_rn(pfr_half_add(x0, x1), x2))), t | (uint32_t(3 * l + 3) << 8));
            take(__fmul_rn(w2, pfr_half_add(x3, pfr_half_add(x1, x2))), t | (uint32_t(3 * l + 2) << 8));
            take(__fmul_rn(w1, __fadd_rn(x2, x3)), t | (uint32_t(3 * l + 1) << 8));
        }
        if (l == 0) take(__fmul_rn(w0, x3), t);
    }
}

template<typename Ts, int L, int DOUT, int l = 0>
__device__ __forceinline__ void pfr_rescan_levels(int winL, const PfWindow<Ts, L, DOUT> &win, float w0, float w1, float w2, float w3, bool full,
                                                  float best, float &val, uint32_t &tok)
{
    if (winL == l) pfr_rescan<Ts, L, DOUT, l>(win, w0, w1, w2, w3, full, best, val, tok);
    if constexpr (l + 1 < L) pfr_rescan_levels<Ts, L, DOUT, l + 1>(winL, win, w0, w1, w2, w3, full, best, val, tok);
}

// Maximum over one level's trials of one output time: x(u), u in [-3 S, ns), in X[u + 3 S].
// POS: largest profile values, multiplied at the end; else every product.
template<int l, int NS, int SS, bool POS>
__device__ __forceinline__ float pfr_group(const float *X, bool full, float w0, float w1, float w2, float w3)
{
    constexpr float NINF = -__builtin_huge_valf();
    float m0 = NINF, m1 = NINF, m2 = NINF, m3 = NINF;   // POS: per profile; else m0 alone
    const float *x = X + 3 * SS;
    if (!full) {
        // width 1: single samples only
#pragma unroll
        for (int u = 0; u < NS; u++) m0 = fmaxf(m0, POS ? x[u] : __fmul_rn(w0, x[u]));
        return POS ? __fmul_rn(w0, m0) : m0;
    }
    float y1[2], y2[2], y3[2];
    float Ap = pfr_half_add(x[-3 * SS], x[-2 * SS]);   // x0/2 + x1; with S = 1 the previous entry's x1/2 + x2
#pragma unroll
    for (int u = 0; u < NS; u++) {
        const float A = pfr_half_add(x[u - 2 * SS], x[u - SS]);
        if (SS > 1 && u > 0) Ap = pfr_half_add(x[u - 3 * SS], x[u - 2 * SS]);
        y1[u & 1] = __fadd_rn(x[u - SS], x[u]);
        y2[u & 1] = pfr_half_add(x[u], A);
        y3[u & 1] = pfr_half_add(x[u], __fadd_rn(Ap, x[u - SS]));
        if (SS == 1) Ap = A;
        if (!POS) {
            y1[u & 1] = __fmul_rn(w1, y1[u & 1]);
            y2[u & 1] = __fmul_rn(w2, y2[u & 1]);
            y3[u & 1] = __fmul_rn(w3, y3[u & 1]);
            m0 = pfr_max3(m0, y1[u & 1], y2[u & 1]);
            m0 = (l == 0) ? pfr_max3(m0, y3[u & 1], __fmul_rn(w0, x[u])) : fmaxf(m0, y3[u & 1]);
        } else if (NS == 1) {
            m0 = x[u];
            m1 = y1[0];
            m2 = y2[0];
            m3 = y3[0];
        } else if (u & 1) {
            if (l == 0) m0 = pfr_max3(m0, x[u - 1], x[u]);
            m1 = pfr_max3(m1, y1[0], y1[1]);
            m2 = pfr_max3(m2, y2[0], y2[1]);
            m3 = pfr_max3(m3, y3[0], y3[1]);
        }
    }
    if (!POS) return m0;
    const float g = pfr_max3(__fmul_rn(w1, m1), __fmul_rn(w2, m2), __fmul_rn(w3, m3));
    return (l == 0) ? fmaxf(g, __fmul_rn(w0, m0)) : g;
}

// One multiplet: own block e, halo block h (level 0 filled), levels l and up. Updates the per-level maxima.
template<typename Ts, int L, int DOUT, bool POS, int l>
__device__ __forceinline__ void pfr_levels(float (&e)[2][DOUT], float (&h)[2][DOUT], int lane, int LW, int base, bool full, const float *wr, int m,
                                           float (&bl)[L], int (&ml)[L])
{
    using R = PfReg<Ts, L, DOUT>;
    constexpr int NS = R::ns(l), SS = R::S(l), CUR = l & 1, NXT = CUR ^ 1;
    // Entries [-3 S, 0) from the lanes before.
    float X[3 * SS + NS];
#pragma unroll
    for (int u = -3 * SS; u < 0; u++) {
        const int q = (-u + NS - 1) / NS, i = u + q * NS;   // q lanes back, entry i
        const float off = (lane >= LW - q) ? h[CUR][i] : e[CUR][i];
        X[u + 3 * SS] = __shfl_sync(0xffffffffu, off, base | ((lane - q) & (LW - 1)));
    }
#pragma unroll
    for (int u = 0; u < NS; u++) X[3 * SS + u] = e[CUR][u];

    const float g = pfr_group<l, NS, SS, POS>(X, full, (l == 0) ? wr[0] : 0.0f, wr[3 * l + 1], wr[3 * l + 2], wr[3 * l + 3]);
    if (g > bl[l]) { bl[l] = g; ml[l] = m; }

    if constexpr (l + 1 < L) {
        if constexpr ((2 << l) <= R::DC) {
#pragma unroll
            for (int u = 0; u < NS / 2; u++) {
                e[NXT][u] = __fadd_rn(e[CUR][2 * u], e[CUR][2 * u + 1]);
                h[NXT][u] = __fadd_rn(h[CUR][2 * u], h[CUR][2 * u + 1]);
            }
        } else {
            // saturated time step: the entry S before, from the same or an earlier lane
#pragma unroll
            for (int u = 0; u < NS; u++) {
                e[NXT][u] = __fadd_rn(X[3 * SS + u - SS], e[CUR][u]);
                float o;
                if (u >= SS) {
                    o = h[CUR][u - SS];
                } else {
                    const int q = (SS - u + NS - 1) / NS, i = u - SS + q * NS;
                    o = __shfl_sync(0xffffffffu, h[CUR][i], base | ((lane - q) & (LW - 1)));
                }
                h[NXT][u] = __fadd_rn(o, h[CUR][u]);
            }
        }
        pfr_levels<Ts, L, DOUT, POS, l + 1>(e, h, lane, LW, base, full, wr, m, bl, ml);
    }
}

template<typename Ts, int L, int DOUT>
__global__ void __launch_bounds__(kPfRegWarps * 32, DOUT <= 16 ? 5 : DOUT == 32 ? 3 : 2) pf_reg_kernel(PfArgs a, int LW)
{
    using R = PfReg<Ts, L, DOUT>;
    constexpr int HL = R::HL, BB = R::BB, NP = 3 * L + 1;
    extern __shared__ __align__(16) unsigned char pfr_sm[];
    const int warp = threadIdx.x >> 5, lane32 = threadIdx.x & 31, G = 32 / LW;
    const int sub = lane32 / LW, lane = lane32 & (LW - 1), base = lane32 & ~(LW - 1);
    const int dm0 = (blockIdx.y * kPfRegWarps + warp) * G;
    const int b = blockIdx.z, bt = a.beam0 + b;
    const int tout0 = blockIdx.x * LW;
    if (dm0 >= a.ndm_out)
        return;   // whole warp exits; warps never synchronize across the block
    // A sub-group past the last coarse dm computes the last one again and stores nothing.
    const bool dm_ok = dm0 + sub < a.ndm_out;
    const int dm = dm_ok ? dm0 + sub : a.ndm_out - 1;
    const int ntw = min(LW, a.nt_out - tout0);
    const int tout = tout0 + min(lane, ntw - 1);
    const int Wds = a.ndm_out / a.ndm_wt, Tds = a.nt_out / a.nt_wt;
    const float *wrow = a.wt + (((long) b * a.ndm_wt + dm / Wds) * a.nt_wt + tout / Tds) * a.P * a.N;
    const Ts *pfrows = (const Ts *) a.pf + ((long) bt * a.ndm_out + dm) * a.M * a.pf_cap;
    const int mask = int(a.pf_cap - 1);
    const bool full = (L > 1) || (a.P > 1);
    const long s0 = a.chunk_ctr ? *a.chunk_ctr * (long) a.nt_chunk : a.s0;
    const int slot0 = int((s0 + (long) tout0 * DOUT) & mask);   // first sample of the warp's first output time

    // NBUF staging buffers per sub-group, of the LW + HL blocks of DOUT samples.
    const int wbytes = (LW + HL) * BB;
    unsigned char *win0 = pfr_sm + (warp * G + sub) * R::NBUF * wbytes;
    const int nch = ((ntw + HL) * BB + 15) / 16;
    auto stage = [&](int m) {
        if (m < a.M) {
            const Ts *row = pfrows + (long) m * a.pf_cap;
            unsigned char *dst = win0 + (m & (R::NBUF - 1)) * wbytes;
            for (int c = lane; c < nch; c += LW)
                cp_async_bytes<16>(dst + 16 * R::swz(c), row + ((slot0 - HL * DOUT + c * int(16 / sizeof(Ts))) & mask));
        }
        cp_async_commit();
    };
#pragma unroll
    for (int m = 0; m < R::NBUF - 1; m++) stage(m);

    float bl[L];
    int ml[L];
#pragma unroll
    for (int l = 0; l < L; l++) { bl[l] = -1.0e30f; ml[l] = 0; }
    float wr[NP];
    int wn = -1;
    bool pos = false;

    for (int m = 0; m < a.M; m++) {
        // Wait for this multiplet's samples (the newer NBUF - 2 may be in flight); then stage another one into the buffer
        // of the previous multiplet, which every lane has read: the iteration ended with a warp barrier.
        cp_async_wait<R::NBUF - 2>();
        __syncwarp();
        stage(m + R::NBUF - 1);
        const int n = a.m_to_n[m];
        if (n != wn) {
            bool ok = true;
#pragma unroll
            for (int p = 0; p < NP; p++) {
                wr[p] = (p < a.P) ? wrow[p * a.N + n] : 1.0f;
                ok = ok && (wr[p] > 0.0f) && (wr[p] < __builtin_huge_valf());
            }
            pos = __all_sync(0xffffffffu, ok);
            wn = n;
        }
        const unsigned char *win = win0 + (m & (R::NBUF - 1)) * wbytes;
        float e[2][DOUT], h[2][DOUT];
        pfr_load<Ts, L, DOUT>(win, HL + lane, e[0]);
        // Halo: the last HL lanes hold the blocks before the first output time, block HL - k in lane LW - k.
        pfr_load<Ts, L, DOUT>(win, max(lane - (LW - HL), 0), h[0]);
        if (pos) pfr_levels<Ts, L, DOUT, true, 0>(e, h, lane, LW, base, full, wr, m, bl, ml);
        else pfr_levels<Ts, L, DOUT, false, 0>(e, h, lane, LW, base, full, wr, m, bl, ml);
        __syncwarp();
    }

    // The first group in the reference's (level, multiplet) order whose maximum is the overall one.
    float best = -1.0e30f;
    int winL = -1, winM = 0;
#pragma unroll
    for (int l = 0; l < L; l++)
        if (bl[l] > best) { best = bl[l]; winL = l; winM = ml[l]; }
    if (lane >= ntw || !dm_ok)
        return;
    float outv = best;
    uint32_t tok = 0xffffffffu;
    if (winL >= 0) {
        const float *w = wrow + a.m_to_n[winM];
        const float w0 = w[0];
        float w1 = 0.0f, w2 = 0.0f, w3 = 0.0f;
        if (full) { w1 = w[(3 * winL + 1) * a.N]; w2 = w[(3 * winL + 2) * a.N]; w3 = w[(3 * winL + 3) * a.N]; }
        PfWindow<Ts, L, DOUT> win;
        win.load(pfrows + (long) winM * a.pf_cap, slot0 + lane * DOUT, mask);
        pfr_rescan_levels<Ts, L, DOUT>(winL, win, w0, w1, w2, w3, full, best, outv, tok);
        tok |= uint32_t(winM) << 16;
    }
    const long o = ((long) b * a.ndm_out + dm) * a.nt_out + tout;
    ((Ts *) a.out_max)[o] = from_f<Ts>(outv);
    a.out_argmax[o] = tok;
}

template<typename Ts, int L, int DOUT>
static void launch_pf_reg(const PfArgs &a, int B, cudaStream_t s)
{
    using R = PfReg<Ts, L, DOUT>;
    // As few lanes per coarse dm as hold a chunk's output times (so that none idles), and the halo.
    int LW = 32;
    while (LW > R::LWMIN && LW / 2 >= a.nt_out) LW /= 2;
    const int G = 32 / LW;
    const size_t sm = (size_t) kPfRegWarps * G * R::NBUF * (LW + R::HL) * R::BB;
    const dim3 grid((a.nt_out + LW - 1) / LW, (a.ndm_out + kPfRegWarps * G - 1) / (kPfRegWarps * G), B);
    set_smem(pf_reg_kernel<Ts, L, DOUT>, sm);
    pf_reg_kernel<Ts, L, DOUT><<<grid, kPfRegWarps * 32, sm, s>>>(a, LW);
    check_launch("pf_reg_kernel");
}

template<typename Ts, int L>
static void launch_pf_reg_d(const PfArgs &a, int B, cudaStream_t s)
{
    switch (a.Dout) {
    case 2: launch_pf_reg<Ts, L, 2>(a, B, s); break;
    case 4: launch_pf_reg<Ts, L, 4>(a, B, s); break;
    case 8: launch_pf_reg<Ts, L, 8>(a, B, s); break;
    case 16: launch_pf_reg<Ts, L, 16>(a, B, s); break;
    case 32: launch_pf_reg<Ts, L, 32>(a, B, s); break;
    case 64: launch_pf_reg<Ts, L, 64>(a, B, s); break;
    default: throw std::runtime_error("pf_reg_kernel: unsupported time downsampling");
    }
}

template<typename Ts>
static void launch_pf_reg_t(const PfArgs &a, int B, cudaStream_t s)
{
    switch (a.L) {
    case 1: launch_pf_reg_d<Ts, 1>(a, B, s); break;
    case 2: launch_pf_reg_d<Ts, 2>(a, B, s); break;
    case 3: launch_pf_reg_d<Ts, 3>(a, B, s); break;
    case 4: launch_pf_reg_d<Ts, 4>(a, B, s); break;
    case 5: launch_pf_reg_d<Ts, 5>(a, B, s); break;
    default: throw std::runtime_error("pf_reg_kernel: unsupported number of boxcar levels");
    }
}

}  // namespace pb2
