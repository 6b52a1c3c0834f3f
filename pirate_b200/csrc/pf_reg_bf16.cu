// pf_reg_bf16.cu -- the register peak finder for bfloat16 storage.

#include "pf_reg.cuh"

namespace pb2 {

void launch_pf_reg_bf16(const PfArgs &a, int B, cudaStream_t s) { launch_pf_reg_t<__nv_bfloat16>(a, B, s); }

}  // namespace pb2
