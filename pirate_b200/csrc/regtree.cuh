// regtree.cuh -- the split of a tree into two register trees, and its sizes (host and device).
//
// A rank-R tree (rows i, butterfly at step r pairs i and i + 2^r with lag bit_reverse(i mod 2^r, r)) is
// computed as two register trees joined by a delay line:
//
//   phase a: rank RA over the low RA row bits (groups f of 2^RA consecutive rows),
//   delay:   row (f, d) of the phase-a output is delayed by P(f, d) = (2^RB - 1 - f) * bit_reverse(d, RA),
//   phase b: rank RB over the high RB row bits (one tree per phase-a output index d).
//
// Shifting a row in time commutes with the butterflies' adds, so every output is the same fp32
// expression of the same inputs as in the one-shot tree (bitwise identical); the phase-b butterfly
// lags reduce to bit_reverse(j, r') < 2^RB. Outputs produced after phase-b step r' of a subband tree
// carry the delay (2^RB - fhi) * bit_reverse(d, RA), which is exactly the subband alignment lag of
// pirate's ReferenceTree (src_lib/ReferenceTree.cpp:41-50), so subband rows come out aligned.
//
// tree_halo.cuh runs the register trees.

#pragma once

#include <cstdint>

namespace pb2 {

__host__ __device__ constexpr int bitrev_c(int x, int n)
{
    int r = 0;
    for (int i = 0; i < n; i++) r = (r << 1) | ((x >> i) & 1);
    return r;
}

// Lag of pair q (0 <= q < 2^(K-1)) at step r of a register tree.
__host__ __device__ constexpr int rt_lag(int r, int q) { return bitrev_c(q & ((1 << r) - 1), r); }

// Staggered subband butterflies of a rank-K phase-b tree at step r: pairs (2k+1, 2k+2) of the
// (K - r)-bit upper index, k < 2^(K-r-1) - 1, for every lower index j < 2^r.
__host__ __device__ constexpr int st_count(int K, int r) { return (K - r - 1 >= 0) ? (((1 << (K - r - 1)) - 1) << r) : 0; }

constexpr int kHaloW = 4;        // samples per thread

// Samples per tile. A tile is 4 bytes of delay line per row and sample; a rank-8 block's rows leave room for 64
// samples, a rank-7 block's for three blocks per SM. Smaller trees take longer tiles, so that a block has at
// least 4 warps and a chunk few barriers.
__host__ __device__ constexpr int halo_tile(int R) { return R >= 7 ? 64 : R == 6 ? 128 : 256; }

__host__ __device__ constexpr int halo_lb4(int F) { return (F + 3) & ~3; }   // lookback F in whole vectors
__host__ __device__ constexpr int halo_len(int F, int delta, int tile) { return halo_lb4(F) + ((F * delta + 3) & ~3) + tile; }

__host__ __device__ constexpr int halo_ring_floats(int RA, int RB)
{
    int o = 0;
    for (int f = 0; f < (1 << RB); f++)
        for (int d = 0; d < (1 << RA); d++) o += halo_len((1 << RB) - 1 - f, bitrev_c(d, RA), halo_tile(RA + RB));
    return o;
}

// Persistent floats per block: the rows' windows without the free tile, then the input rows' last samples
// (sized for 32-bit storage).
__host__ __device__ constexpr long halo_state_floats(int RA, int RB)
{
    return halo_ring_floats(RA, RB) - halo_tile(RA + RB) * (1 << (RA + RB)) + (1 << (RA + RB)) * 16;
}

}  // namespace pb2
