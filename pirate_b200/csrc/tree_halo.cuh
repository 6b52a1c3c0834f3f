// tree_halo.cuh -- the two-phase tree without shuffles: every thread computes a whole register tree over
// a short run of samples, reading the earlier samples that the tree's lags reach back to ("halo") from
// shared memory instead of exchanging intermediate rows with other lanes.
//
// A rank-R tree is split as in regtree.cuh (phase a: rank RA over the low row bits, a delay of
// P(f, d) = F * brev(d) samples with F = 2^RB - 1 - f, phase b: rank RB over the high row bits). Work is
// done in tiles of halo_tile(R) samples, kHaloW consecutive samples of a group of rows per thread:
//
//   - Phase a: a thread loads its kHaloW samples of the group's 2^RA rows and, for row i, the 2^RA - 1 - i
//     samples before them, runs the tree in registers (the partial sums of the halo are recomputed: 88 adds
//     more than the 256 of a rank-4 tree) and stores the outputs at their delayed time u = t + P(f, d).
//   - Phase b: the same with the 2^RB rows of one d, all at one time, so its loads are 16-byte aligned.
//
// A partial sum recomputed by two threads is the same fp32 expression of the same samples, so the
// results are bitwise those of the butterflies with kept histories, and a block's state is the input
// samples and phase-a rows that the next chunk reaches back to.
//
// What bounds it: instruction issue and the shared-memory pipe together. A rank-8 block fills an SM's shared memory,
// so 8 warps have to hide the loads' latency with the trees' own parallelism (about 200 registers per thread);
// measured on stage 1, 23 thread instructions per row and sample, issue 43% active, shared pipe 64%. The form with a
// lane per sample, shuffled lags and kept histories executed 60. Four rank-16 beams, fp16, five trees, 2048 samples:
// stage 1 1.99 -> 1.26 ms, stage 2 2.39 -> 1.49 ms; sixteen rank-12 beams, three trees: 0.49 -> 0.23 and 0.61 ->
// 0.24 ms. kHaloW = 4: the halo costs a third of a rank-4 tree's adds at 4 samples and half as much at 8, but 8 would
// leave a rank-8 block 4 warps.
//
// Alignment is known at compile time everywhere. Phase a's input rows start at sample p with
// p mod 4 = ((i + 1) * dm) mod 4 for a block-wide dm (stage 2; aligned in stage 1): four instances of the
// code. Phase a's unaligned stores: a warp's 4 groups have distinct F mod 4, so for odd brev(d) the 32
// lanes of a scalar store fall on distinct banks, and rows with brev(d) even are stored as 8- or 16-byte
// vectors, which are aligned.
//
// The delay line between the phases is one shared-memory buffer for all rows: row r's window
// [T - lb4, T + P + tile) of delayed times u lies at A_r + lb4 + u, the windows back to back, and all windows
// advance together by one tile, each into the samples its successor has just dropped. So no index wraps: the
// buffer has room for HaloDims::SEG samples of that, and a longer chunk is done in segments that start again at
// T = 0 from the saved state.

#pragma once

#include "devutil.cuh"
#include "regtree.cuh"

#include <type_traits>

namespace pb2 {

// Window offsets A_r of row r = f * 2^RA + d; A[2^(RA+RB)] = M.
template<int RA, int RB>
struct HaloTab
{
    int A[(1 << (RA + RB)) + 1];
};
template<int RA, int RB>
__host__ __device__ constexpr HaloTab<RA, RB> make_halo_tab()
{
    HaloTab<RA, RB> t{};
    int o = 0;
    for (int f = 0; f < (1 << RB); f++)
        for (int d = 0; d < (1 << RA); d++) {
            t.A[(f << RA) + d] = o;
            o += halo_len((1 << RB) - 1 - f, bitrev_c(d, RA), halo_tile(RA + RB));
        }
    t.A[1 << (RA + RB)] = o;
    return t;
}
// Samples kept before a tile's input rows: 2^RA - 1, in whole 16-byte chunks of EPC samples.
__host__ __device__ constexpr int halo_lbk(int RA, int EPC) { return ((1 << RA) - 1 + EPC - 1) / EPC * EPC; }

// Time ranges of a rank-K register tree computed by one thread: after 'level' steps row i is needed over
// [lo, hi), the outputs over [0, W).
template<int K, int W>
struct HaloExt
{
    int lo[K + 1][1 << K], hi[K + 1][1 << K];
};
template<int K, int W>
__host__ __device__ constexpr HaloExt<K, W> make_halo_ext()
{
    HaloExt<K, W> e{};
    for (int i = 0; i < (1 << K); i++) { e.lo[K][i] = 0; e.hi[K][i] = W; }
    for (int r = K - 1; r >= 0; r--)
        for (int i0 = 0; i0 < (1 << K); i0++) {
            if (i0 & (1 << r)) continue;
            const int i1 = i0 | (1 << r), L = bitrev_c(i0 & ((1 << r) - 1), r);
            const int a0 = e.lo[r + 1][i0], b0 = e.hi[r + 1][i0], a1 = e.lo[r + 1][i1], b1 = e.hi[r + 1][i1];
            e.lo[r][i1] = a0 < a1 ? a0 : a1;
            e.hi[r][i1] = b0 > b1 ? b0 : b1;
            e.lo[r][i0] = a0 - L < a1 - L - 1 ? a0 - L : a1 - L - 1;
            e.hi[r][i0] = b0 - L > b1 - L - 1 ? b0 - L : b1 - L - 1;
        }
    return e;
}

// The same for phase b of a subband tree: the rows after every step are outputs themselves, and the odd bands
// (but the last) are also the lower halves of the staggered pairs (2k + 1, 2k + 2).
template<int K, int W>
__host__ __device__ constexpr HaloExt<K, W> make_halo_ext_sub()
{
    HaloExt<K, W> e{};
    for (int i = 0; i < (1 << K); i++) { e.lo[K][i] = 0; e.hi[K][i] = W; }
    for (int r = K - 1; r >= 0; r--)
        for (int i0 = 0; i0 < (1 << K); i0++) {
            if (i0 & (1 << r)) continue;
            const int i1 = i0 | (1 << r), L = bitrev_c(i0 & ((1 << r) - 1), r);
            const int a0 = e.lo[r + 1][i0], a1 = e.lo[r + 1][i1];
            e.lo[r][i1] = a0 < a1 ? a0 : a1;
            if (i1 < (1 << K) - (1 << r) && e.lo[r][i1] > -L - 1) e.lo[r][i1] = -L - 1;
            e.lo[r][i0] = a0 - L < a1 - L - 1 ? a0 - L : a1 - L - 1;
            e.hi[r][i0] = e.hi[r][i1] = W;
        }
    return e;
}

// Two fp32 additions in one sm_100 packed f32x2 instruction, each rounded to nearest.
__device__ __forceinline__ float2 halo_add2(float2 a, float2 b)
{
    unsigned long long x, y, d;
    asm("mov.b64 %0, {%1, %2};" : "=l"(x) : "f"(a.x), "f"(a.y));
    asm("mov.b64 %0, {%1, %2};" : "=l"(y) : "f"(b.x), "f"(b.y));
    asm("add.rn.f32x2 %0, %1, %2;" : "=l"(d) : "l"(x), "l"(y));
    float2 r;
    asm("mov.b64 {%0, %1}, %2;" : "=f"(r.x), "=f"(r.y) : "l"(d));
    return r;
}

// Index of sample 0 in a row's registers: even, so that even samples start register pairs.
__host__ __device__ constexpr int halo_org(int K) { return K > 0 ? (1 << K) : 2; }

// n[t] = butterfly of x[t - L] and y[t] for t in [lo, hi): even lags two samples at a time.
template<bool NORM, int W, int O>
__device__ __forceinline__ void halo_add(float (&n)[W + O], const float (&x)[W + O], const float (&y)[W + O], int L, int lo, int hi)
{
#pragma unroll
    for (int t = -O; t < W; t += 2) {
        const bool a = (t >= lo && t < hi), b = (t + 1 >= lo && t + 1 < hi);
        if (a && b && (L & 1) == 0) {
            const float2 s = halo_add2(make_float2(x[t - L + O], x[t + 1 - L + O]), make_float2(y[t + O], y[t + 1 + O]));
            n[t + O] = NORM ? __fmul_rn(kRsqrt2, s.x) : s.x;
            n[t + 1 + O] = NORM ? __fmul_rn(kRsqrt2, s.y) : s.y;
        } else {
            if (a) n[t + O] = bfly_n<NORM>(x[t - L + O], y[t + O]);
            if (b) n[t + 1 + O] = bfly_n<NORM>(x[t + 1 - L + O], y[t + 1 + O]);
        }
    }
}

// Rows [BASE, BASE + 2^LV) of the tree through their first LV steps, depth first (upper half, lower half,
// then the step that joins them), which keeps the live registers close to the outputs'. load(row) fills
// v[row][t + O] over the input range. Sample t of a row is v[row][t + O].
template<int K, int W, bool NORM, int LV, int BASE, typename Load>
__device__ __forceinline__ void halo_tree(float (&v)[1 << K][W + halo_org(K)], Load load)
{
    constexpr HaloExt<K, W> E = make_halo_ext<K, W>();
    constexpr int O = halo_org(K);
    if constexpr (LV == 0) {
        load(std::integral_constant<int, BASE>(), std::integral_constant<int, E.lo[0][BASE]>(),
             std::integral_constant<int, E.hi[0][BASE]>());
    } else {
        constexpr int h = 1 << (LV - 1);
        halo_tree<K, W, NORM, LV - 1, BASE + h>(v, load);
        halo_tree<K, W, NORM, LV - 1, BASE>(v, load);
#pragma unroll
        for (int j = 0; j < h; j++) {
            const int i0 = BASE + j, i1 = BASE + j + h, L = bitrev_c(j, LV - 1);
            float n0[W + O], n1[W + O];
            halo_add<NORM, W, O>(n0, v[i0], v[i1], L, E.lo[LV][i0], E.hi[LV][i0]);
            halo_add<NORM, W, O>(n1, v[i0], v[i1], L + 1, E.lo[LV][i1], E.hi[LV][i1]);
#pragma unroll
            for (int t = -O; t < W; t++) {
                if (t >= E.lo[LV][i0] && t < E.hi[LV][i0]) v[i0][t + O] = n0[t + O];
                if (t >= E.lo[LV][i1] && t < E.hi[LV][i1]) v[i1][t + O] = n1[t + O];
            }
        }
    }
}

// Four consecutive samples from an address aligned to four samples.
template<typename Ts>
__device__ __forceinline__ void halo_load4(const Ts *p, float (&o)[4])
{
    if constexpr (sizeof(Ts) == 4) {
        const float4 q = *(const float4 *) p;
        o[0] = q.x; o[1] = q.y; o[2] = q.z; o[3] = q.w;
    } else {
        const uint2 q = *(const uint2 *) p;
        const uint32_t w[2] = {q.x, q.y};
#pragma unroll
        for (int i = 0; i < 2; i++) {
            float2 f;
            if constexpr (std::is_same<Ts, __half>::value) {
                f = __half22float2(*(const __half2 *) &w[i]);
            } else {
                const uint32_t a = w[i] << 16, b = w[i] & 0xffff0000u;
                f = make_float2(*(const float *) &a, *(const float *) &b);
            }
            o[2 * i] = f.x;
            o[2 * i + 1] = f.y;
        }
    }
}

template<typename Ts>
__device__ __forceinline__ void halo_store4(Ts *p, const float (&o)[4])
{
    if constexpr (sizeof(Ts) == 4) {
        *(float4 *) p = make_float4(o[0], o[1], o[2], o[3]);
    } else {
        uint2 q;
        if constexpr (std::is_same<Ts, __half>::value) {
            const __half2 a = __floats2half2_rn(o[0], o[1]), b = __floats2half2_rn(o[2], o[3]);
            q.x = *(const uint32_t *) &a;
            q.y = *(const uint32_t *) &b;
        } else {
            const __nv_bfloat162 a = __floats2bfloat162_rn(o[0], o[1]), b = __floats2bfloat162_rn(o[2], o[3]);
            q.x = *(const uint32_t *) &a;
            q.y = *(const uint32_t *) &b;
        }
        *(uint2 *) p = q;
    }
}

// Block geometry and shared-memory layout.
template<typename Ts_, int RA_, int RB_, int STAGE_>
struct HaloDims
{
    using Ts = Ts_;
    static constexpr int RA = RA_, RB = RB_, STAGE = STAGE_;
    static constexpr int NA = 1 << RA, NB = 1 << RB, NR = NA * NB;
    static constexpr int TILE = halo_tile(RA + RB), TL = TILE / kHaloW;   // samples and threads per group and tile
    static constexpr int NT = NA * TL;                            // threads: one phase-b run each
    static constexpr int NW = NT / 32, RPW = NR / NW;             // warps, input rows per warp
    // Samples per segment: 2048 where shared memory allows, less where it costs a block per SM.
    static constexpr int SEG = (RA + RB == 8) ? (sizeof(Ts) == 4 ? 1024 : 2048) : (RA + RB == 7) ? (sizeof(Ts) == 4 ? 2048 : 512) : 2048;
    static constexpr int EPC = 16 / sizeof(Ts);                   // samples per 16-byte chunk
    static constexpr int LBK = halo_lbk(RA, EPC);
    static constexpr int SPR = LBK + TILE + (STAGE == 2 ? EPC : 0);       // samples per staged row
    // Groups of rows start 64 bytes apart modulo 128, so that two groups' 8-byte loads share no bank.
    static constexpr int GSTR = NA * SPR + (((64 - NA * SPR * int(sizeof(Ts))) % 128 + 128) % 128) / int(sizeof(Ts));
    static constexpr int M = halo_ring_floats(RA, RB);
    static constexpr bool NORM = (sizeof(Ts) == 4);
    static constexpr int SU = NORM ? 0 : RA + RB;                 // unnormalized steps of an output
    static constexpr size_t tabw = 0;                             // int[NR]: phase-a store offsets, [f][d]
    static constexpr size_t tabr = tabw + 4 * NR;                 // int[NR]: phase-b load offsets, [d][f]
    static constexpr int PARTS = TILE / 32, PSTR = NR + 8;        // 8: a warp's parts lie in different banks
    static constexpr size_t outpos = tabr + 4 * NR;               // int[PARTS][PSTR]: stage 1, output positions, [d][f]
    static constexpr size_t in_tab = tabr + 4 * NR;               // int4[NR]: stage 2, input rows
    static constexpr size_t stg = (tabr + 4 * NR + (STAGE == 1 ? 4 * PARTS * PSTR : 16 * NR) + 127) & ~size_t(127);
    static constexpr size_t ring = (stg + sizeof(Ts) * GSTR * NB + 127) & ~size_t(127);
    static constexpr size_t total = ring + 4 * (M + SEG - TILE);  // the last tile of a segment starts at SEG - TILE
    static_assert(total <= 232448, "shared memory per block");
    static_assert(RPW >= 1 && RPW * NW == NR, "rows per warp");
    // Blocks per SM that shared memory and a register budget (168 per thread with 16-row trees, 80 below) allow; rank-6
    // stage 2 runs 2 blocks at 112 registers rather than 3 at 80 (16 rank-12 beams, fp16: 0.280 -> 0.242 ms), rank-6
    // stage 1 3 (0.224 ms against 0.235).
    static constexpr int fit = int(233472 / (total + 1024)), rfit = 65536 / ((RB == 4 ? 168 : RB == 3 && STAGE == 2 ? 112 : 80) * NT);
    static constexpr int MINB = fit < rfit ? (fit < 1 ? 1 : fit) : (rfit < 1 ? 1 : rfit);
};

// Entry i of a table row of N ints (16-byte loads where the row is a multiple of 16 bytes).
template<int N>
__device__ __forceinline__ int halo_tab(const int *row, int i)
{
    if constexpr (N % 4 != 0) {
        return row[i];
    } else {
        const int4 t = ((const int4 *) row)[i >> 2];
        return (i & 3) == 0 ? t.x : (i & 3) == 1 ? t.y : (i & 3) == 2 ? t.z : t.w;
    }
}

// Offset of staged row r (group f = r / NA), in samples.
template<class D> __device__ __forceinline__ int halo_row(int r) { return (r >> D::RA) * D::GSTR + (r & (D::NA - 1)) * D::SPR; }

// Stage-2 input rows start at sample p of their delay lines, p mod 8 = ((r + 1) dm) mod 8 with the block's
// dm; DM4 = dm mod 4 fixes the shift within a vector at compile time, and bit 2 of p is that of
// ((i + 1) DM4) mod 8 xor t, with t one of two block constants by the parity of i + 1 (xor f * dm in 4-row
// groups).
//
// Phase a of one tile of 'tile' samples at T by thread 'tid'; ring: the delay line at T.
template<class D, int DM4>
__device__ __forceinline__ void halo_phase_a(int tid, int tile, int dm, const typename D::Ts *stg, float *ring, const int *tabw)
{
    constexpr int NA = D::NA, NB = D::NB, RA = D::RA, O = halo_org(RA);
    const int warp = tid >> 5, lane = tid & 31;
    constexpr int TQ = (NB >= 4) ? D::TL / 8 : D::TL / 16;      // a warp covers 4 groups x 8 runs, or 2 x 16
    constexpr int NC = (NB >= 4) ? NB / 4 * TQ : TQ;
    for (int c = warp; c < NC; c += D::NW) {
        const int f = (NB >= 4) ? 4 * (c / TQ) + (lane >> 3) : (lane >> 4);
        const int tl = (NB >= 4) ? 8 * (c % TQ) + (lane & 7) : 16 * c + (lane & 15);
        if (kHaloW * tl >= tile) continue;
        const typename D::Ts *base = stg + f * D::GSTR + D::LBK + kHaloW * tl;
        // Offsets of the rows whose start has bit 2 of the constant part clear (0) or set (1).
        int off[2][2] = {{0, 0}, {0, 0}};
        if constexpr (D::STAGE == 2 && D::EPC == 8) {
            const int te = (NA == 4) ? (f & dm & 1) : 0, to = te ^ ((dm >> 2) & 1);
            off[0][0] = 4 * te; off[0][1] = 4 - 4 * te;
            off[1][0] = 4 * to; off[1][1] = 4 - 4 * to;
        }
        float v[NA][kHaloW + O];
        halo_tree<RA, kHaloW, D::NORM, RA, 0>(v, [&](auto I, auto LO, auto HI) {
            constexpr int i = decltype(I)::value, lo = decltype(LO)::value, hi = decltype(HI)::value;
            if constexpr (D::STAGE == 2 && RA < 2) {
                // one- and two-row groups: the shift depends on the group, so single samples at run time
                const int r = f * NA + i;
                const typename D::Ts *p = base + i * D::SPR + (((r + 1 - D::NR) * dm) & (D::EPC - 1));
#pragma unroll
                for (int t = lo; t < hi; t++) v[i][t + O] = to_f(p[t]);
            } else {
                constexpr int cc = ((i + 1) * DM4) & 7, s = cc & 3;
                const typename D::Ts *p = base + i * D::SPR;
                if constexpr (D::STAGE == 2 && D::EPC == 8) p += off[(i + 1) & 1][cc >> 2];
                constexpr int b0 = (s + lo + 64) / 4 - 16, b1 = (s + hi - 1 + 64) / 4 - 16;
#pragma unroll
                for (int b = b0; b <= b1; b++) {
                    float q[4];
                    halo_load4(p + 4 * b, q);
#pragma unroll
                    for (int e = 0; e < 4; e++) {
                        const int t = 4 * b + e - s;
                        if (t >= lo && t < hi) v[i][t + O] = q[e];
                    }
                }
            }
        });
        const int *tw = tabw + f * NA;
        float *rt = ring + kHaloW * tl;
#pragma unroll
        for (int d = 0; d < NA; d++) {
            const int delta = bitrev_c(d, RA);
            float *w = rt + halo_tab<NA>(tw, d);
            const float x[4] = {v[d][O], v[d][O + 1], v[d][O + 2], v[d][O + 3]};
            if (delta % 4 == 0) {
                *(float4 *) w = make_float4(x[0], x[1], x[2], x[3]);
            } else if (delta % 2 == 0) {
                *(float2 *) w = make_float2(x[0], x[1]);
                *(float2 *) (w + 2) = make_float2(x[2], x[3]);
            } else {
#pragma unroll
                for (int k = 0; k < 4; k++) w[k] = x[k];
            }
        }
    }
}

// Phase b of one tile by thread 'tid': thread (d, tl); emit(f, x) takes output row f's 4 samples.
template<class D, typename Emit>
__device__ __forceinline__ void halo_phase_b(int tid, int tile, const float *ring, const int *tabr, Emit emit)
{
    constexpr int NB = D::NB, RB = D::RB, O = halo_org(RB);
    const int d = tid / D::TL, tl = tid % D::TL;
    if (kHaloW * tl >= tile) return;
    float v[NB][kHaloW + O];
    halo_tree<RB, kHaloW, D::NORM, RB, 0>(v, [&](auto I, auto LO, auto HI) {
        constexpr int f = decltype(I)::value, lo = decltype(LO)::value, hi = decltype(HI)::value;
        constexpr int lb = halo_lb4(NB - 1 - f);
        const float *p = ring + halo_tab<NB>(tabr + d * NB, f) + kHaloW * tl;
#pragma unroll
        for (int b = 0; b <= lb / 4; b++) {
            const float4 q4 = *(const float4 *) (p + 4 * b);
            const float q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int t = 4 * b + e - lb;
                if (t >= lo && t < hi) v[f][t + O] = q[e];
            }
        }
    });
#pragma unroll
    for (int f = 0; f < NB; f++) {
        const float x[4] = {tree_out(v[f][O], D::SU), tree_out(v[f][O + 1], D::SU), tree_out(v[f][O + 2], D::SU),
                            tree_out(v[f][O + 3], D::SU)};
        emit(f, x);
    }
}

// Phase b of a subband tree (FrequencySubbands multiplet order, ReferenceTree::dedisperse_2d,
// src_lib/ReferenceTree.cpp:120-300): rows of peak-finding level 0 are phase b's inputs, level r + 1 the outputs
// of step r: even band pairs are the in-place butterflies, odd ("staggered") pairs (2k + 1, 2k + 2) extra ones.
// cnt[l] bands and first multiplet mb[l] per level; emit(m, x) takes multiplet m's 4 samples.
template<class D, typename Emit>
__device__ __forceinline__ void halo_phase_b_sub(int tid, int tile, const float *ring, const int *tabr, const int *cnt, const int *mb, Emit emit)
{
    constexpr int NB = D::NB, RB = D::RB, O = halo_org(RB), W = kHaloW;
    constexpr int SA = D::NORM ? 0 : D::RA;
    constexpr HaloExt<RB, W> E = make_halo_ext_sub<RB, W>();
    const int d = tid / D::TL, tl = tid % D::TL;
    if (W * tl >= tile) return;
    float v[NB][W + O];
#pragma unroll
    for (int f = 0; f < NB; f++) {
        const int lb = halo_lb4(NB - 1 - f);
        const float *p = ring + halo_tab<NB>(tabr + d * NB, f) + W * tl;
#pragma unroll
        for (int b = 0; b <= halo_lb4(NB - 1) / 4; b++) {
            if (4 * b > lb || 4 * b + 3 - lb < E.lo[0][f]) continue;
            const float4 q4 = *(const float4 *) (p + 4 * b);
            const float q[4] = {q4.x, q4.y, q4.z, q4.w};
#pragma unroll
            for (int e = 0; e < 4; e++) {
                const int t = 4 * b + e - lb;
                if (t >= E.lo[0][f] && t < W) v[f][t + O] = q[e];
            }
        }
    }
    if (cnt[0] > 0) {
#pragma unroll
        for (int f = 0; f < NB; f++)
            if (f < cnt[0]) {
                const float x[4] = {tree_out(v[f][O], SA), tree_out(v[f][O + 1], SA), tree_out(v[f][O + 2], SA), tree_out(v[f][O + 3], SA)};
                emit(mb[0] + f, x);
            }
    }
#pragma unroll
    for (int r = 0; r < RB; r++) {
        const int h = 1 << r, c = cnt[r + 1], m0 = mb[r + 1], S = SA + (D::NORM ? 0 : r + 1);
        if (c >= 2) {
#pragma unroll
            for (int u = 0; u < st_count(RB, r); u++) {
                const int k = u >> r, j = u & (h - 1), L = rt_lag(r, j);
                const int qa = ((2 * k + 1) << r) | j, qb = ((2 * k + 2) << r) | j;
                if (2 * k + 1 < c) {
                    float x[4], y[4];
#pragma unroll
                    for (int t = 0; t < W; t++) {
                        x[t] = tree_out(bfly_n<D::NORM>(v[qa][t - L + O], v[qb][t + O]), S);
                        y[t] = tree_out(bfly_n<D::NORM>(v[qa][t - L - 1 + O], v[qb][t + O]), S);
                    }
                    const int m = m0 + (2 * k + 1) * (2 << r) + 2 * bitrev_c(j, r);
                    emit(m, x);
                    emit(m + 1, y);
                }
            }
        }
#pragma unroll
        for (int q = 0; q < NB / 2; q++) {
            const int i0 = ((q >> r) << (r + 1)) | (q & (h - 1)), i1 = i0 + h, L = rt_lag(r, q);
            float n0[W + O], n1[W + O];
            halo_add<D::NORM, W, O>(n0, v[i0], v[i1], L, E.lo[r + 1][i0], W);
            halo_add<D::NORM, W, O>(n1, v[i0], v[i1], L + 1, E.lo[r + 1][i1], W);
#pragma unroll
            for (int t = -O; t < W; t++) {
                if (t >= E.lo[r + 1][i0]) v[i0][t + O] = n0[t + O];
                if (t >= E.lo[r + 1][i1]) v[i1][t + O] = n1[t + O];
            }
        }
        if (c > 0) {
#pragma unroll
            for (int q = 0; q < NB / 2; q++) {
                const int i0 = ((q >> r) << (r + 1)) | (q & (h - 1)), k = q >> r, j = q & (h - 1);
                if (2 * k < c) {
                    const int m = m0 + (2 * k) * (2 << r) + 2 * bitrev_c(j, r);
                    const float x[4] = {tree_out(v[i0][O], S), tree_out(v[i0][O + 1], S), tree_out(v[i0][O + 2], S), tree_out(v[i0][O + 3], S)};
                    const float y[4] = {tree_out(v[i0 + h][O], S), tree_out(v[i0 + h][O + 1], S), tree_out(v[i0 + h][O + 2], S), tree_out(v[i0 + h][O + 3], S)};
                    emit(m, x);
                    emit(m + 1, y);
                }
            }
        }
    }
}

}  // namespace pb2
