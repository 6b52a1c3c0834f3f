// devutil.cuh -- device helpers shared by the dedispersion kernels: storage conversions, butterflies,
// asynchronous copies.

#pragma once

#include <cstdint>
#include <stdexcept>
#include <string>

#include <cuda_bf16.h>
#include <cuda_fp16.h>
#include <cuda_runtime.h>

namespace pb2 {

constexpr float kRsqrt2 = 0.7071067811865476f;

template<typename T> __host__ __device__ __forceinline__ float to_f(T x);
template<> __host__ __device__ __forceinline__ float to_f<float>(float x) { return x; }
template<> __host__ __device__ __forceinline__ float to_f<__half>(__half x) { return __half2float(x); }
template<> __host__ __device__ __forceinline__ float to_f<__nv_bfloat16>(__nv_bfloat16 x) { return __bfloat162float(x); }

template<typename T> __device__ __forceinline__ T from_f(float x);
template<> __device__ __forceinline__ float from_f<float>(float x) { return x; }
template<> __device__ __forceinline__ __half from_f<__half>(float x) { return __float2half_rn(x); }
template<> __device__ __forceinline__ __nv_bfloat16 from_f<__nv_bfloat16>(float x) { return __float2bfloat16_rn(x); }

__device__ __forceinline__ float bfly(float x, float y) { return __fmul_rn(kRsqrt2, __fadd_rn(x, y)); }

// Tree butterflies with (NORM) or without the per-step 1/sqrt2. float32 storage normalizes at every
// step, as the reference does, so that its outputs are bitwise the reference's. 16-bit storage keeps
// its in-register fp32 sums unnormalized and scales once, by tree_scale(steps) = 2^(-steps/2), where a
// value leaves the registers (a stored row or an emitted subband): one rounding instead of one per
// step, and one multiply per stored value instead of one per butterfly.
template<bool NORM>
__device__ __forceinline__ float bfly_n(float x, float y) { return NORM ? bfly(x, y) : __fadd_rn(x, y); }

__host__ __device__ constexpr float tree_scale(int steps)
{
    float s = (steps & 1) ? kRsqrt2 : 1.0f;
    for (int i = 0; i < steps / 2; i++) s *= 0.5f;
    return s;
}

// A value leaving the registers after n unnormalized butterflies (n is a compile-time constant at
// every call site once the step loops are unrolled).
__device__ __forceinline__ float tree_out(float v, int n) { return n ? __fmul_rn(v, tree_scale(n)) : v; }

__device__ __forceinline__ int brev_bits(int x, int nbits) { return nbits ? int(__brev(unsigned(x)) >> (32 - nbits)) : 0; }

template<int BYTES>
__device__ __forceinline__ void cp_async_bytes(void *smem, const void *gmem)
{
    unsigned s = (unsigned) __cvta_generic_to_shared(smem);
    asm volatile("cp.async.ca.shared.global [%0], [%1], %2;\n" :: "r"(s), "l"(gmem), "n"(BYTES) : "memory");
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template<int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" :: "n"(N) : "memory"); }
__device__ __forceinline__ void cp_async_wait0() { asm volatile("cp.async.wait_group 0;\n" ::: "memory"); }

inline void check_launch(const char *what)
{
    cudaError_t e = cudaGetLastError();
    if (e != cudaSuccess)
        throw std::runtime_error(std::string(what) + ": " + cudaGetErrorString(e));
}

template<typename K>
inline void set_smem(K kernel, size_t bytes)
{
    cudaError_t e = cudaFuncSetAttribute(kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int) bytes);
    if (e != cudaSuccess) throw std::runtime_error(std::string("cudaFuncSetAttribute: ") + cudaGetErrorString(e));
}

}  // namespace pb2
