// tree_halo_f16.cu -- the halo tree kernels for float16 storage.

#include "tree_halo_kernel.cuh"

namespace pb2 {

void launch_stage1_halo_f16(const Stage1Args &a, int nblocks, int B, cudaStream_t s)
{
    launch_halo_t<__half, 1, false>(a, a.rank, nblocks, B, s);
}

void launch_stage2_halo_f16(const Stage2Multi &m, bool sub, int nblocks, int B, cudaStream_t s)
{
    if (sub) launch_halo_t<__half, 2, true>(m, m.t[0].rank, nblocks, B, s);
    else launch_halo_t<__half, 2, false>(m, m.t[0].rank, nblocks, B, s);
}

}  // namespace pb2
