// pf_reg_main_f16.cu -- the register peak finder for float16 storage, widths to 32 and a time downsampling of 16.

#include "pf_reg.cuh"

namespace pb2 {

template<> void launch_pf_reg_5_16<__half>(const PfArgs &a, int B, cudaStream_t s) { launch_pf_reg<__half, 5, 16>(a, B, s); }

}  // namespace pb2
