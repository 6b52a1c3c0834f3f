// tree_halo_kernel.cuh -- the tree kernels of stage 1 and stage 2 on tree_halo.cuh's register trees. Compiled
// once per storage type (tree_halo_f32.cu, tree_halo_f16.cu, tree_halo_bf16.cu), in parallel.

#pragma once

#include "kernels.cuh"
#include "tree_halo.cuh"

#include <algorithm>
#include <cstring>
#include <stdexcept>
#include <string>
#include <type_traits>

namespace pb2 {

template<int RA, int RB> __constant__ HaloTab<RA, RB> c_halo_tab = make_halo_tab<RA, RB>();

template<int STAGE> struct HaloParamOf;
template<> struct HaloParamOf<1> { using type = Stage1Args; };
template<> struct HaloParamOf<2> { using type = Stage2Multi; };
template<int STAGE> struct HaloArgsOf;
template<> struct HaloArgsOf<1> { using type = Stage1Args; };
template<> struct HaloArgsOf<2> { using type = Stage2Args; };

template<int STAGE, typename PT>
__device__ __forceinline__ const typename HaloArgsOf<STAGE>::type &halo_args(const PT &P, int ti)
{
    if constexpr (STAGE == 1) return P;
    else return P.t[ti];
}

// One block per (tree block, beam); see tree_halo.cuh. Per tile: barrier (this tile's input staged, the
// previous tile's phase b done), phase a, barrier, then the next tile's copies are issued and overlap
// phase b.
//   STAGE 1: input = level-p tree rows (aligned), output = per-row stage-1 delay lines.
//   STAGE 2: input = stage-1 delay lines read at lag rb_lag (misaligned), output = subband rows (SUB) or the
//            full band's only.
template<typename Ts, int RA, int RB, int STAGE, bool SUB>
__global__ void __launch_bounds__(HaloDims<Ts, RA, RB, STAGE>::NT, SUB ? 1 : HaloDims<Ts, RA, RB, STAGE>::MINB)
tree_halo_kernel(const __grid_constant__ typename HaloParamOf<STAGE>::type P)
{
    using D = HaloDims<Ts, RA, RB, STAGE>;
    constexpr int NA = D::NA, NB = D::NB, NR = D::NR, EPC = D::EPC, LBK = D::LBK, TILE = D::TILE, TL = D::TL;
    // Stage 2: this block's tree ti and its block index blk among that tree's nblk blocks.
    int ti = 0, blk = blockIdx.x, nblk = gridDim.x;
    if constexpr (STAGE == 2) {
        while (ti + 1 < P.n && blk >= P.blk0[ti + 1]) ti++;
        nblk = P.blk0[ti + 1] - P.blk0[ti];
        blk -= P.blk0[ti];
    }
    const auto &a = halo_args<STAGE>(P, ti);
    extern __shared__ __align__(128) unsigned char sm_raw[];
    int *tabw = (int *) (sm_raw + D::tabw), *tabr = (int *) (sm_raw + D::tabr), *outpos = (int *) (sm_raw + D::outpos);
    int4 *in_tab = (int4 *) (sm_raw + D::in_tab);
    Ts *stg = (Ts *) (sm_raw + D::stg);
    float *ring0 = (float *) (sm_raw + D::ring);

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int b = blockIdx.y, bt = a.beam0 + b;
    const long s0 = a.chunk_ctr ? *a.chunk_ctr * (long) a.nt : a.s0;
    // Tiles of TILE samples, the last one of what remains (a multiple of 32). (Equal tiles, of the largest power of two
    // that divides the chunk, took up to 8% longer on chunks of other lengths.)
    const int ntiles = (a.nt + TILE - 1) / TILE;
    float *st = a.state + ((long) bt * nblk + blk) * a.state_per_block;
    Ts *st_in = (Ts *) (st + (D::M - TILE * NR));
    const HaloTab<RA, RB> &tab = c_halo_tab<RA, RB>;
    const int row0 = warp * D::RPW;   // this warp's input rows and state rows

    // The rows' windows at T = 0 from the state, or at T to the state.
    auto load_windows = [&]() {
        for (int r = row0; r < row0 + D::RPW; r++) {
            const int A = tab.A[r], n = tab.A[r + 1] - A - TILE;
            for (int j = 4 * lane; j < n; j += 128) cp_async_bytes<16>(ring0 + A + j, st + A - TILE * r + j);
        }
    };
    auto save_windows = [&](int T) {
        for (int r = row0; r < row0 + D::RPW; r++) {
            const int A = tab.A[r], n = tab.A[r + 1] - A - TILE;
            for (int j = 4 * lane; j < n; j += 128)
                *(float4 *) (st + A - TILE * r + j) = *(const float4 *) (ring0 + A + T + j);
        }
    };
    load_windows();
    if constexpr (LBK > 0)
        for (int i = lane; i < D::RPW * (LBK / EPC); i += 32) {
            const int r = row0 + i / (LBK / EPC), k = i % (LBK / EPC);
            cp_async_bytes<16>(stg + halo_row<D>(r) + k * EPC, st_in + r * LBK + k * EPC);
        }

    const Ts *in;
    int pos1 = 0, dm = 0;               // stage 1: read position of every input row; stage 2: the rows' lag factor
    int opos = 0, oend = 0, ocap = 0;   // stage 1: output line [d][f] = tid (next position, end, capacity)
    Ts *out = nullptr;
    if constexpr (STAGE == 1) {
        in = (const Ts *) a.in + (long) (a.in_beam0 + b) * a.in_beam_stride + (long) blk * NR * a.in_row_stride;
        pos1 = int(((a.chunk_ctr && a.in_mask != -1) ? s0 : a.in_s0) & a.in_mask);
        out = (Ts *) a.ring + (long) bt * a.ring_beam_stride + a.ring_off[(long) blk * NR];
    } else {
        in = (const Ts *) a.ring + (long) bt * a.ring_beam_stride;
        dm = brev_bits(blk, a.amb_rank) + (a.uflag ? (1 << a.amb_rank) : 0);
    }
    for (int r = tid; r < NR; r += D::NT) {
        const int f = r >> RA, d = r & (NA - 1), F = NB - 1 - f, A = tab.A[r];
        tabw[r] = A + halo_lb4(F) + F * brev_bits(d, RA);
        tabr[d * NB + f] = A;
    }
    // Positions of the tile's parts of 32 samples in this thread's output line. Lines hold a multiple of 32 samples, so no
    // part wraps; a position per tile would need lines of whole tiles or chunks, up to twice the memory for a chunk that
    // is no multiple of the tile.
    auto next_outpos = [&]() {
#pragma unroll
        for (int j = 0; j < D::PARTS; j++) {
            outpos[j * D::PSTR + tid] = opos;
            opos = (opos + 32 == oend) ? oend - ocap : opos + 32;
        }
    };
    if constexpr (STAGE == 1) {
        static_assert(D::NT >= NR, "one thread per output line");
        if (tid < NR) {
            // the host checks that a block's lines span < 2^31 samples
            const long row = (long) blk * NR + ((tid % NB) << RA) + tid / NB;
            const int off = int(a.ring_off[row] - a.ring_off[(long) blk * NR]);
            ocap = a.ring_cap[row];
            opos = off + int(s0 % ocap);
            oend = off + ocap;
        }
    } else {
        for (int r = row0 + lane; r < row0 + D::RPW; r += 32) {
            const long row = ((long) r << a.amb_rank) + blk;
            const long lag = (long) (NR - 1 - r) * dm, cap = a.ring_cap[row], off = a.ring_off[row];
            const long p = (s0 - lag) % cap;
            in_tab[r] = make_int4(int(p < 0 ? p + cap : p), int(cap), int(off & 0xffffffffL), int(off >> 32));
        }
        __syncwarp();
    }

    // Copies the next tile of this warp's input rows behind their lookback, 16 bytes per copy, consecutive
    // lanes on consecutive chunks of a row.
    constexpr int NCH = TILE / EPC;   // chunks per whole tile
    auto issue = [&](int next) {
        const int ch = min(TILE, a.nt - next * TILE) / EPC;
        if constexpr (STAGE == 1) {
            for (int i = lane; i < D::RPW * NCH; i += 32) {
                const int r = row0 + i / NCH, k = i % NCH;
                if (k < ch)
                    cp_async_bytes<16>(stg + halo_row<D>(r) + LBK + k * EPC, in + (long) r * a.in_row_stride + ((pos1 + k * EPC) & a.in_mask));
            }
            pos1 = int((pos1 + TILE) & a.in_mask);
        } else {
            // One chunk more than the tile, from p & ~(EPC - 1); capacities are multiples of 32 samples, so a
            // chunk never straddles the end of a line and wraps at most once.
            auto copy = [&](int r, int k) {
                const int4 t = in_tab[r];
                int q = (t.x & ~(EPC - 1)) + k * EPC;
                q = (q >= t.y) ? q - t.y : q;
                cp_async_bytes<16>(stg + halo_row<D>(r) + LBK + k * EPC, in + ((long) t.w << 32 | (unsigned) t.z) + q);
            };
            for (int i = lane; i < D::RPW * NCH; i += 32)
                if (i % NCH < ch) copy(row0 + i / NCH, i % NCH);
            for (int r = row0 + lane; r < row0 + D::RPW; r += 32) copy(r, ch);
            __syncwarp();
            for (int r = row0 + lane; r < row0 + D::RPW; r += 32) {
                const int4 t = in_tab[r];
                const int x = t.x + TILE;
                in_tab[r].x = (x >= t.y) ? x - t.y : x;
            }
            __syncwarp();
        }
        cp_async_commit();
    };
    issue(0);

    // Stage 2: multiplet 0 of this thread's coarse dm (d = tid / TL), at its samples of the tile.
    Ts *pf_rows = nullptr;
    int pf_slot = 0;
    if constexpr (STAGE == 2) {
        const int pf_dm = brev_bits(tid / TL, RA);
        const long rowbase = ((long) bt * a.ndm_out + ((long) brev_bits(blk, a.amb_rank) << RA) + pf_dm) * a.M;
        pf_rows = (Ts *) a.pf + rowbase * a.pf_cap;
        pf_slot = int(s0 & (a.pf_cap - 1));
    }

    int T = 0;   // of the segment
    for (int it = 0; it < ntiles; it++) {
        if (T == D::SEG) {
            // Next segment: the windows move back to T = 0 through the state (each thread reloads what it saved).
            __syncthreads();
            save_windows(T);
            __syncthreads();
            load_windows();
            cp_async_commit();
            T = 0;
        }
        const int len = min(TILE, a.nt - it * TILE);
        float *ring = ring0 + T;
        cp_async_wait0();
        __syncthreads();
        if constexpr (STAGE == 1) {
            if (tid < NR) next_outpos();
            halo_phase_a<D, 0>(tid, len, 0, stg, ring, tabw);
        } else {
            switch (RA < 2 ? 0 : dm & 3) {
            case 0: halo_phase_a<D, 0>(tid, len, dm, stg, ring, tabw); break;
            case 1: halo_phase_a<D, 1>(tid, len, dm, stg, ring, tabw); break;
            case 2: halo_phase_a<D, 2>(tid, len, dm, stg, ring, tabw); break;
            default: halo_phase_a<D, 3>(tid, len, dm, stg, ring, tabw); break;
            }
        }
        __syncthreads();
        // The next tile's lookback: the last LBK samples before its first chunk.
        if constexpr (LBK > 0) {
            constexpr int NV = D::RPW * (LBK / EPC), PL = (NV + 31) / 32;
            uint4 x[PL];
#pragma unroll
            for (int j = 0; j < PL; j++) {
                const int i = lane + 32 * j;
                if (i < NV) x[j] = *(const uint4 *) (stg + halo_row<D>(row0 + i / (LBK / EPC)) + len + i % (LBK / EPC) * EPC);
            }
#pragma unroll
            for (int j = 0; j < PL; j++) {
                const int i = lane + 32 * j;
                if (i < NV) *(uint4 *) (stg + halo_row<D>(row0 + i / (LBK / EPC)) + i % (LBK / EPC) * EPC) = x[j];
            }
            __syncwarp();
        }
        if (it + 1 < ntiles) issue(it + 1);
        if constexpr (STAGE == 1) {
            constexpr int PV = 32 / kHaloW;   // threads per part
            Ts *o = out + kHaloW * (tid % PV);
            const int *op = outpos + (tid % TL / PV) * D::PSTR + (tid / TL) * NB;
            halo_phase_b<D>(tid, len, ring, tabr, [&](int f, const float (&x)[4]) { halo_store4(o + halo_tab<NB>(op, f), x); });
        } else {
            Ts *o = pf_rows + ((pf_slot + kHaloW * (tid % TL)) & int(a.pf_cap - 1));
            auto emit = [&](int m, const float (&x)[4]) { halo_store4(o + (long) m * a.pf_cap, x); };
            if constexpr (SUB) {
                halo_phase_b_sub<D>(tid, len, ring, tabr, a.sb_count, a.sb_mbase, emit);
            } else {
                halo_phase_b<D>(tid, len, ring, tabr, [&](int f, const float (&x)[4]) {
                    // the full band's multiplet of output row f
                    emit(2 * bitrev_c(f & (NB / 2 - 1), RB - 1) + (f >= NB / 2 ? 1 : 0), x);
                });
            }
            pf_slot = int((pf_slot + TILE) & (a.pf_cap - 1));
        }
        T += len;
    }

    // Windows and lookback back to the state (the windows are only read in phase b, the lookback is this
    // warp's own).
    save_windows(T);
    if constexpr (LBK > 0)
        for (int i = lane; i < D::RPW * (LBK / EPC); i += 32) {
            const int r = row0 + i / (LBK / EPC), k = i % (LBK / EPC);
            *(uint4 *) (st_in + r * LBK + k * EPC) = *(const uint4 *) (stg + halo_row<D>(r) + k * EPC);
        }
}

template<typename Ts, int R, int STAGE, bool SUB, typename A>
static void launch_halo_r(const A &a, int nblocks, int B, cudaStream_t s)
{
    constexpr int RA = split_ra(R), RB = split_rb(R);
    using D = HaloDims<Ts, RA, RB, STAGE>;
    set_smem(tree_halo_kernel<Ts, RA, RB, STAGE, SUB>, D::total);
    tree_halo_kernel<Ts, RA, RB, STAGE, SUB><<<dim3(nblocks, B), D::NT, D::total, s>>>(a);
    check_launch(STAGE == 1 ? "stage1 tree_halo_kernel" : "stage2 tree_halo_kernel");
}

template<typename Ts, int STAGE, bool SUB, typename A>
static void launch_halo_t(const A &a, int rank, int nblocks, int B, cudaStream_t s)
{
    switch (rank) {
    case 1: launch_halo_r<Ts, 1, STAGE, SUB>(a, nblocks, B, s); break;
    case 2: launch_halo_r<Ts, 2, STAGE, SUB>(a, nblocks, B, s); break;
    case 3: launch_halo_r<Ts, 3, STAGE, SUB>(a, nblocks, B, s); break;
    case 4: launch_halo_r<Ts, 4, STAGE, SUB>(a, nblocks, B, s); break;
    case 5: launch_halo_r<Ts, 5, STAGE, SUB>(a, nblocks, B, s); break;
    case 6: launch_halo_r<Ts, 6, STAGE, SUB>(a, nblocks, B, s); break;
    case 7: launch_halo_r<Ts, 7, STAGE, SUB>(a, nblocks, B, s); break;
    case 8: launch_halo_r<Ts, 8, STAGE, SUB>(a, nblocks, B, s); break;
    default: throw std::runtime_error("tree_halo_kernel: unsupported dd rank " + std::to_string(rank));
    }
}

}  // namespace pb2
