// FP64 velocity moments of distributions, and the macroscopic fields made of
// them (frfs/plugins/dgfsmomwriterstd.py:14-313).
#include "common.cuh"
#include "rows.cuh"

namespace bdgfs {

// cell-centre velocities: in the launch's parameters (Nv <= kMaxNv), or on the device
struct MomentGrid {
    double v[kMaxNv];
    const double* dev;
};

struct MomentOut {
    double *raw;                        // [ndof][13], or the five fields below
    double *rho, *U, *T, *q, *P;        // [ndof], [3], [1], [3], [6]
};

constexpr int kMomThreads = 128, kMom = 13;

// rho, U, T, q, P of raw moments m = (f, c f, c c f (xx xy xz yy yz zz),
// |c|^2 c f): P_ab = 2 sum (c-U)_a (c-U)_b f, T = (2/3) sum |c-U|^2 f / rho,
// q_a = sum |c-U|^2 (c-U)_a f
__device__ __forceinline__ void macro_store(const double (&m)[kMom], const MomentOut& o, int64_t dof)
{
    const double rho = m[0];
    const double U[3] = {m[1] / rho, m[2] / rho, m[3] / rho};
    const double S[3][3] = {{m[4], m[5], m[6]}, {m[5], m[7], m[8]}, {m[6], m[8], m[9]}};
    double P[6];
    int k = 0;
#pragma unroll
    for (int a = 0; a < 3; ++a)
#pragma unroll
        for (int b = a; b < 3; ++b) P[k++] = 2.0 * (S[a][b] - rho * U[a] * U[b]);
    const double trS = S[0][0] + S[1][1] + S[2][2];
    const double U2 = U[0] * U[0] + U[1] * U[1] + U[2] * U[2];
    const double Um = U[0] * m[1] + U[1] * m[2] + U[2] * m[3];
    o.rho[dof] = rho;
    o.T[dof] = (P[0] + P[3] + P[5]) / 2.0 * (2.0 / 3.0) / rho;
#pragma unroll
    for (int a = 0; a < 3; ++a) {
        o.U[3 * dof + a] = U[a];
        o.q[3 * dof + a] = m[10 + a] - trS * U[a] - 2.0 * (S[a][0] * U[0] + S[a][1] * U[1] + S[a][2] * U[2])
                           + 2.0 * U[a] * Um + U2 * m[1 + a] - (rho * U2) * U[a];
    }
#pragma unroll
    for (int j = 0; j < 6; ++j) o.P[6 * dof + j] = P[j];
}

// One CTA per distribution.  A thread takes VEC consecutive z of one (x, y)
// line and keeps their four z-sums (f, cz f, cz^2 f, cz^3 f); the 13 moments
// follow from those with 16 more multiply-adds per chunk, so an element costs
// 4 + 16/VEC FP64 operations and one conversion instead of 13 and three 64-bit
// index divisions.  Bound: shared memory (the coordinates: 82 % of its wavefronts),
// then the FP64 pipe (54 %) and HBM (each row read once: 0.63 of the copy rate).  Measured
// with the fields formed in the same launch (they were some 30 small ones):
// 5670 rows of 24^3 FP32 834 -> 74 us, 4.2 TB/s; 256 threads and one element
// each was the form before.
template <typename T, int VEC, int NVC, bool MACRO>
__global__ void __launch_bounds__(kMomThreads) moments_kernel(const T* __restrict__ f, int Nvr, const MomentGrid g,
                                                              double cw, const MomentOut o)
{
    extern __shared__ double cs[];                     // [Nv]
    __shared__ double red[kMom][kMomThreads + 1];
    const int Nv = NVC > 0 ? NVC : Nvr;
    const uint32_t n = uint32_t(Nv) * Nv * Nv;
    const int64_t dof = blockIdx.x;
    const T* row = f + dof * int64_t(n);
    for (int i = threadIdx.x; i < Nv; i += kMomThreads) cs[i] = g.dev ? g.dev[i] : g.v[i];
    __syncthreads();
    double m[kMom];
#pragma unroll
    for (int j = 0; j < kMom; ++j) m[j] = 0.0;
#pragma unroll 2
    for (uint32_t v = threadIdx.x * VEC; v < n; v += kMomThreads * VEC) {
        T x[VEC];
        if constexpr (VEC >= 4 && sizeof(T) == 4) {
#pragma unroll
            for (int j = 0; j < VEC; j += 4) {
                const float4 w = __ldcs(reinterpret_cast<const float4*>(row + v + j));
                x[j] = w.x; x[j + 1] = w.y; x[j + 2] = w.z; x[j + 3] = w.w;
            }
        } else if constexpr (VEC >= 2) {
#pragma unroll
            for (int j = 0; j < VEC; j += 2) {
                const double2 w = __ldcs(reinterpret_cast<const double2*>(row + v + j));
                x[j] = w.x; x[j + 1] = w.y;
            }
        } else {
            x[0] = __ldcs(row + v);
        }
        uint32_t ix, iy, iz;
        vsplit<NVC>(v, uint32_t(Nv), ix, iy, iz);
        const double cx = cs[ix], cy = cs[iy];
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
#pragma unroll
        for (int j = 0; j < VEC; ++j) {
            const double cz = cs[iz + j];
            double t = double(x[j]);
            s0 += t;
            t *= cz;
            s1 += t;
            t *= cz;
            s2 += t;
            s3 = fma(t, cz, s3);
        }
        const double a = cx * s0, b = cy * s0, c2 = fma(cx, cx, cy * cy), e = fma(c2, s0, s2);
        m[0] += s0;
        m[1] += a;
        m[2] += b;
        m[3] += s1;
        m[4] = fma(cx, a, m[4]);
        m[5] = fma(cx, b, m[5]);
        m[6] = fma(cx, s1, m[6]);
        m[7] = fma(cy, b, m[7]);
        m[8] = fma(cy, s1, m[8]);
        m[9] += s2;
        m[10] = fma(cx, e, m[10]);
        m[11] = fma(cy, e, m[11]);
        m[12] += fma(c2, s1, s3);
    }
#pragma unroll
    for (int j = 0; j < kMom; ++j) red[j][threadIdx.x] = m[j];
    __syncthreads();
    // each warp sums every fourth row; lane 0 leaves the sum in column 0
    const int lane = threadIdx.x & 31;
    for (int j = threadIdx.x >> 5; j < kMom; j += kMomThreads / 32) {
        double s = (red[j][lane] + red[j][lane + 32]) + (red[j][lane + 64] + red[j][lane + 96]);
#pragma unroll
        for (int k = 16; k > 0; k >>= 1) s += __shfl_xor_sync(0xffffffffu, s, k);
        __syncwarp();
        if (lane == 0) red[j][0] = s * cw;
    }
    __syncthreads();
    if constexpr (MACRO) {
        if (threadIdx.x == 0) {
#pragma unroll
            for (int j = 0; j < kMom; ++j) m[j] = red[j][0];
            macro_store(m, o, dof);
        }
    } else if (threadIdx.x < kMom) {
        o.raw[dof * kMom + threadIdx.x] = red[threadIdx.x][0];
    }
}

template <typename T, int VEC, bool MACRO>
static int moments_nv(const T* f, int64_t ndof, int Nv, const MomentGrid& g, double cw, const MomentOut& o,
                      cudaStream_t st)
{
    const size_t smem = size_t(Nv) * sizeof(double);
#define GO(NN) moments_kernel<T, VEC, NN, MACRO><<<unsigned(ndof), kMomThreads, smem, st>>>(f, Nv, g, cw, o)
    if (VEC == 8 && Nv == 16) GO((VEC == 8 ? 16 : 0));
    else if (VEC == 8 && Nv == 24) GO((VEC == 8 ? 24 : 0));
    else if (VEC == 8 && Nv == 32) GO((VEC == 8 ? 32 : 0));
    else GO(0);
#undef GO
    return cuda_status(cudaGetLastError());
}

// eight z per thread when they share a line and the rows are 16-byte aligned
// (four where Nv has only that factor), else one
template <typename T, bool MACRO>
static int moments_launch(const void* f, int64_t ndof, int Nv, const MomentGrid& g, double cw, const MomentOut& o,
                          cudaStream_t st)
{
    const T* p = static_cast<const T*>(f);
    const bool al = (reinterpret_cast<uintptr_t>(f) & 15u) == 0;
    if (al && Nv % 8 == 0) return moments_nv<T, 8, MACRO>(p, ndof, Nv, g, cw, o, st);
    if (al && Nv % 4 == 0) return moments_nv<T, 4, MACRO>(p, ndof, Nv, g, cw, o, st);
    return moments_nv<T, 1, MACRO>(p, ndof, Nv, g, cw, o, st);
}

}  // namespace bdgfs

using namespace bdgfs;

// velocity index in 32 bits, c0 in shared memory
static bool moments_ok(int64_t ndof, int32_t Nv) { return ndof >= 0 && ndof <= 2147483647LL && Nv >= 1 && Nv <= 1600; }

extern "C" int32_t bdgfs_moments(const void* f, int64_t ndof, int32_t Nv, int32_t fp64, const double* c0, double cw,
                                 double* out, void* stream)
{
    if (!f || !c0 || !out || !moments_ok(ndof, Nv)) return BDGFS_EINVAL;
    if (ndof == 0) return BDGFS_OK;
    MomentGrid g{};
    g.dev = c0;
    MomentOut o{};
    o.raw = out;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return fp64 ? moments_launch<double, false>(f, ndof, Nv, g, cw, o, st)
                : moments_launch<float, false>(f, ndof, Nv, g, cw, o, st);
}

extern "C" int32_t bdgfs_macroscopic(const void* f, int64_t ndof, int32_t Nv, int32_t fp64, const double* c0_host,
                                     double cw, double* rho, double* U, double* T, double* q, double* P,
                                     void* stream)
{
    if (!f || !c0_host || !rho || !U || !T || !q || !P || !moments_ok(ndof, Nv) || Nv > kMaxNv) return BDGFS_EINVAL;
    if (ndof == 0) return BDGFS_OK;
    MomentGrid g{};
    for (int i = 0; i < Nv; ++i) g.v[i] = c0_host[i];
    const MomentOut o{nullptr, rho, U, T, q, P};
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    return fp64 ? moments_launch<double, true>(f, ndof, Nv, g, cw, o, st)
                : moments_launch<float, true>(f, ndof, Nv, g, cw, o, st);
}
