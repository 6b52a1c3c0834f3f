// pf_reg_f32.cu -- the register peak finder for float32 storage.

#include "pf_reg.cuh"

namespace pb2 {

void launch_pf_reg_f32(const PfArgs &a, int B, cudaStream_t s) { launch_pf_reg_t<float>(a, B, s); }

}  // namespace pb2
