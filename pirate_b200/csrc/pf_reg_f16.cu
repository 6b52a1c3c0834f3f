// pf_reg_f16.cu -- the register peak finder for float16 storage.

#include "pf_reg.cuh"

namespace pb2 {

void launch_pf_reg_f16(const PfArgs &a, int B, cudaStream_t s) { launch_pf_reg_t<__half>(a, B, s); }

}  // namespace pb2
