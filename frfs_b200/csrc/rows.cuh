// Per-distribution row helpers shared by the hybrid and BGK kernels: one
// CTA walks one velocity cube f[v], v = (ix*Nv + iy)*Nv + iz.
#pragma once
#include <cstdint>

namespace bdgfs {

constexpr int kMaxNv = 64;

// velocity index v = (ix*Nv + iy)*Nv + iz, 32-bit arithmetic; NVC > 0: Nv
// known at compile time (the divisions become multiplications)
template <int NVC = 0>
__device__ __forceinline__ void vsplit(uint32_t v, uint32_t Nv, uint32_t& ix, uint32_t& iy, uint32_t& iz)
{
    const uint32_t N = NVC > 0 ? uint32_t(NVC) : Nv;
    const uint32_t q = v / N;
    iz = v - q * N;
    ix = q / N;
    iy = q - ix * N;
}

// Four consecutive values (same x, y; z..z+3) of a row: one 16-byte load
// for float, two for double (VEC = 4), or one scalar (VEC = 1).
template <typename T, int VEC>
struct Chunk {
    T v[VEC];
    __device__ __forceinline__ void load(const T* p)
    {
        if constexpr (VEC == 4 && sizeof(T) == 4) {
            const float4 x = *reinterpret_cast<const float4*>(p);
            v[0] = x.x; v[1] = x.y; v[2] = x.z; v[3] = x.w;
        } else if constexpr (VEC == 4) {
            const double2 a = reinterpret_cast<const double2*>(p)[0];
            const double2 b = reinterpret_cast<const double2*>(p)[1];
            v[0] = a.x; v[1] = a.y; v[2] = b.x; v[3] = b.y;
        } else {
            v[0] = *p;
        }
    }
    __device__ __forceinline__ void store(T* p) const
    {
        if constexpr (VEC == 4 && sizeof(T) == 4) {
            *reinterpret_cast<float4*>(p) = make_float4(v[0], v[1], v[2], v[3]);
        } else if constexpr (VEC == 4) {
            reinterpret_cast<double2*>(p)[0] = make_double2(v[0], v[1]);
            reinterpret_cast<double2*>(p)[1] = make_double2(v[2], v[3]);
        } else {
            *p = v[0];
        }
    }
};

// Walk of a row in steps of a fixed number of values: the index split kept by
// carries instead of two divisions per step.  step < Nv^3.
struct RowWalk {
    uint32_t ix, iy, iz, dx, dy, dz, N;
    __device__ __forceinline__ RowWalk(uint32_t v, uint32_t step, uint32_t Nv) : N(Nv)
    {
        vsplit(v, Nv, ix, iy, iz);
        vsplit(step, Nv, dx, dy, dz);
    }
    __device__ __forceinline__ void next()
    {
        iz += dz;
        iy += dy;
        ix += dx;
        if (iz >= N) { iz -= N; ++iy; }
        if (iy >= N) { iy -= N; ++ix; }
    }
};

// FP64 moments of a chunk added to m: {1, c, |c|^2} (NA = 5), then {cx^2, cy^2,
// cz^2, cx cy, cy cz, cz cx} (NA = 11), then {|c|^2 c} (NA = 14).  The chunk's
// z-sums (of x, cz x, cz^2 x, cz^3 x) come first, so a value costs one
// conversion and 3 or 4 FP64 operations and the rest is per chunk.
template <typename T, int VEC, int NA>
__device__ __forceinline__ void chunk_moments(const Chunk<T, VEC>& c, double cx, double cy, const double* cz,
                                              double (&m)[NA])
{
    static_assert(NA == 5 || NA == 11 || NA == 14, "5, 11 or 14 moment rows");
    // every rounding written out: kernels that reduce the same row in the same
    // order get the same bits, however the compiler contracts
    double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
    for (int j = 0; j < VEC; ++j) {
        const double z = cz[j];
        double t = double(c.v[j]);
        s0 = __dadd_rn(s0, t);
        t = __dmul_rn(t, z);
        s1 = __dadd_rn(s1, t);
        if constexpr (NA == 14) {
            t = __dmul_rn(t, z);
            s2 = __dadd_rn(s2, t);
            s3 = fma(t, z, s3);
        } else {
            s2 = fma(t, z, s2);
        }
    }
    const double a = __dmul_rn(cx, s0), b = __dmul_rn(cy, s0), r2 = fma(cx, cx, __dmul_rn(cy, cy));
    const double e = fma(r2, s0, s2);
    m[0] = __dadd_rn(m[0], s0);
    m[1] = __dadd_rn(m[1], a);
    m[2] = __dadd_rn(m[2], b);
    m[3] = __dadd_rn(m[3], s1);
    m[4] = __dadd_rn(m[4], e);
    if constexpr (NA >= 11) {
        m[5] = fma(cx, a, m[5]);
        m[6] = fma(cy, b, m[6]);
        m[7] = __dadd_rn(m[7], s2);
        m[8] = fma(cx, b, m[8]);
        m[9] = fma(cy, s1, m[9]);
        m[10] = fma(cx, s1, m[10]);
    }
    if constexpr (NA == 14) {
        m[11] = fma(cx, e, m[11]);
        m[12] = fma(cy, e, m[12]);
        m[13] = __dadd_rn(m[13], fma(r2, s1, s3));
    }
}

// FP64 raw moments {sum x, sum c x, sum |c|^2 x} of one row (block-wide)
template <typename T, int VEC>
__device__ __forceinline__ void row_moments(const T* __restrict__ row, int n, int Nv, const double* cs,
                                            double (&m)[5])
{
#pragma unroll 2
    for (int v = threadIdx.x * VEC; v < n; v += blockDim.x * VEC) {
        Chunk<T, VEC> c;
        c.load(row + v);
        uint32_t ix, iy, iz;
        vsplit(uint32_t(v), uint32_t(Nv), ix, iy, iz);
        chunk_moments<T, VEC, 5>(c, cs[ix], cs[iy], cs + iz, m);
    }
}

}  // namespace bdgfs
