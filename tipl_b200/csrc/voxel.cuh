// Voxels of every storage type as floats, and float order as integer order.
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace regb {

// DT: the codes of regb_dtype.  Integers become floats on the ALU and FP pipes (the bits of
// 2^23 + v, minus 2^23: both steps exact), not in the conversion unit.
template <int DT>
__device__ __forceinline__ float load_as_float(const void* p, long long i);
template <>
__device__ __forceinline__ float load_as_float<0>(const void* p, long long i)
{
    return __fsub_rn(__uint_as_float(0x4B000000u | ((const uint8_t*)p)[i]), 8388608.0f);
}
template <>
__device__ __forceinline__ float load_as_float<1>(const void* p, long long i)
{
    return ((const float*)p)[i];
}
template <>
__device__ __forceinline__ float load_as_float<2>(const void* p, long long i)
{
    return __fsub_rn(__uint_as_float(0x4B000000u | ((const uint16_t*)p)[i]), 8388608.0f);
}
template <>
__device__ __forceinline__ float load_as_float<3>(const void* p, long long i)
{
    return __uint_as_float((unsigned)((const uint16_t*)p)[i] << 16);
}

// Order-preserving integer key of a float (for atomicMin/atomicMax).
__device__ __forceinline__ unsigned key_of(float f)
{
    const unsigned u = __float_as_uint(f);
    return (u & 0x80000000u) ? ~u : (u | 0x80000000u);
}
// and back
__device__ __forceinline__ float float_of(unsigned k)
{
    return __uint_as_float((k & 0x80000000u) ? (k & 0x7fffffffu) : ~k);
}

}  // namespace regb
