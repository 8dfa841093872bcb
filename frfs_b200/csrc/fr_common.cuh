// Velocity-row helpers of the FR kernels.
#pragma once
#include "common.cuh"

namespace bdgfs {

// velocity components of index v
template <typename T>
__device__ __forceinline__ void vel(const T* c0, int Nv, int64_t v, T (&c)[3])
{
    // v < Nv^3 <= 2^18: 32-bit arithmetic
    const uint32_t vv = uint32_t(v), n = uint32_t(Nv);
    const uint32_t q = vv / n, iz = vv - q * n;
    const uint32_t ix = q / n, iy = q - ix * n;
    c[0] = c0[ix];
    c[1] = c0[iy];
    c[2] = c0[iz];
}

// VB consecutive values of a velocity row (one vector access when aligned)
template <typename T, int VB>
struct Vec {
    T v[VB];
    __device__ __forceinline__ void load(const T* __restrict__ p)
    {
        if constexpr (VB == 4 && sizeof(T) == 4) {
            const float4 x = *reinterpret_cast<const float4*>(p);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        } else if constexpr (VB == 2 && sizeof(T) == 4) {
            const float2 x = *reinterpret_cast<const float2*>(p);
            v[0] = x.x; v[1] = x.y;
        } else if constexpr (VB == 2 && sizeof(T) == 8) {
            const double2 x = *reinterpret_cast<const double2*>(p);
            v[0] = x.x; v[1] = x.y;
        } else {
#pragma unroll
            for (int q = 0; q < VB; ++q) v[q] = p[q];
        }
    }
    __device__ __forceinline__ void store(T* __restrict__ p) const
    {
        if constexpr (VB == 4 && sizeof(T) == 4) {
            *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        } else if constexpr (VB == 2 && sizeof(T) == 4) {
            *reinterpret_cast<float2*>(p) = make_float2(v[0], v[1]);
        } else if constexpr (VB == 2 && sizeof(T) == 8) {
            *reinterpret_cast<double2*>(p) = make_double2(v[0], v[1]);
        } else {
#pragma unroll
            for (int q = 0; q < VB; ++q) p[q] = v[q];
        }
    }
};

// first velocity of the chunk of VB velocities that holds the mirror
// images of v0 .. v0 + VB - 1 under c_d -> -c_d (the grid is symmetric:
// c0[Nv - 1 - i] = -c0[i]); for the z axis the chunk holds them reversed.
// Chunks never straddle a z line (VB divides Nv when a y or z mirror is
// in use, checked on the host).
__device__ __forceinline__ int64_t mirror_chunk(int64_t v0, int Nv, int kind, int VB)
{
    const int64_t N = Nv, N2 = N * N;
    if (kind == BDGFS_BC_SPECULAR_X) return v0 + (N - 1 - 2 * (v0 / N2)) * N2;
    if (kind == BDGFS_BC_SPECULAR_Y) return v0 + (N - 1 - 2 * ((v0 / N) % N)) * N;
    const int64_t iz = v0 % N;
    return v0 - iz + (N - iz - VB);
}

// VB velocities per thread when every row is VB-aligned
template <typename T>
static int vec_width(int64_t nv, const void* const* ptrs, int n, int VB = sizeof(T) == 4 ? 4 : 2)
{
    if (nv % VB) return 1;
    for (int i = 0; i < n; ++i)
        if (ptrs[i] && (reinterpret_cast<uintptr_t>(ptrs[i]) % (VB * sizeof(T)))) return 1;
    return VB;
}

}  // namespace bdgfs
