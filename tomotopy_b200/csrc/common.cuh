// common.cuh -- small device helpers and host error types shared by the
// engine's translation units.
#pragma once
#include <cuda_runtime.h>
#include <cstdint>
#include <stdexcept>
#include <string>

namespace tmtk {

constexpr unsigned FULL = 0xFFFFFFFFu;

__device__ __forceinline__ float hs_scan32(float x, int lane)
{
#pragma unroll
    for (int off = 1; off < 32; off <<= 1) {
        const float y = __shfl_up_sync(FULL, x, off);
        if (lane >= off) x = __fadd_rn(x, y);
    }
    return x;
}

// one Hillis-Steele step: lanes below `off` keep x
__device__ __forceinline__ float hs_up(float x, int off)
{
    float r;
    asm volatile("{\n .reg .pred p;\n .reg .f32 y;\n"
                 " shfl.sync.up.b32 y|p, %1, %2, 0, 0xffffffff;\n"
                 " mov.f32 %0, %1;\n"
                 " @p add.rn.f32 %0, %1, y;\n}"
                 : "=&f"(r) : "f"(x), "r"(off));
    return r;
}

// the value of the lane before, 0 in lane 0
__device__ __forceinline__ float up1_or_0(float x)
{
    float r;
    asm volatile("{\n .reg .pred p;\n .reg .f32 y;\n"
                 " shfl.sync.up.b32 y|p, %1, 1, 0, 0xffffffff;\n"
                 " selp.f32 %0, y, 0f00000000, p;\n}"
                 : "=f"(r) : "f"(x));
    return r;
}

// 1 / x rounded to nearest, without a branch, for x in [2^-107, 2^104): one Newton step
// from an approximation within one ulp is exact rounding but for divisors whose
// mantissa is all ones (P. Markstein, "Computation of elementary functions on the IBM
// RISC System/6000 processor", IBM J. Res. Dev. 34, 1990), where it depends on the
// approximation; on sm_100 it equals __frcp_rn for every mantissa of these
// exponents (tests/test_recip_gpu.py).
__device__ __forceinline__ float recip_mid(float x)
{
    float y;
    asm("rcp.approx.ftz.f32 %0, %1;" : "=f"(y) : "f"(x));
    return __fmaf_rn(y, __fmaf_rn(-x, y, 1.f), y);
}

__host__ __device__ __forceinline__ uint32_t round4(uint32_t x) { return (x + 3u) & ~3u; }

__device__ __forceinline__ double warp_sum(double x)
{
#pragma unroll
    for (int o = 16; o; o >>= 1) x += __shfl_xor_sync(FULL, x, o);
    return x;
}

struct CudaError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
struct ArgError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
struct OomError : std::runtime_error {
    using std::runtime_error::runtime_error;
};
struct StateError : std::runtime_error {
    using std::runtime_error::runtime_error;
};

#define CK(call)                                                                              \
    do {                                                                                      \
        cudaError_t e_ = (call);                                                              \
        if (e_ != cudaSuccess)                                                                \
            throw CudaError(std::string(#call) + ": " + cudaGetErrorString(e_));              \
    } while (0)


} // namespace tmtk
