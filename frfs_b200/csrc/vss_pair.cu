// Mixture VSS collision operator for two species at Nv = 24, FP32, with an
// antipodal direction set: Q_p = sum_q Q_pq (vss.cu states the operator and the
// reference).
//
// For a direction s and its opposite the slices repeat: with a -> -a the two
// factors of T_pq(s) = IFFT(e^{+i mu_q a} F_p) IFFT(e^{-i mu_p a} F_q) are those of
// T_qp, so T_qp(-s) = T_pq(s) and T_pp(-s) = T_pp(s), exactly.  One radius then
// needs M/2 slices for each species with itself and M for the unlike pair,
// whose transform feeds both gains, instead of 4 M; the kernel weights of s and
// -s are added in the table (their sum is real: b(-s) = conj b(s)).
//
// One persistent CTA of 320 threads per distribution (or per range of radii of
// one, when distributions are few).  A slice carries its two factors as the two
// lanes of f32x2 numbers through the inverse passes x, y, z, multiplies them in
// registers, and transforms the product z, y, x.  The exchange cube holds
// (A.re, B.re, A.im, B.im) at (x*24 + y)*25 + z: every pass reads and writes its
// own pencils in place, in 16-byte accesses free of bank conflicts; the product
// goes into the same rows as 8-byte numbers, offset by one in every second
// group of eight rows.  G^ of both species stays in tensor memory.  F comes from
// the CTA's scratch and the weights from their tables, through L2: 165 KB (like
// pair) or 442 KB a slice.  Measured on one B200, Nrho = M = 12, 370 argon-krypton
// pairs: 25.6 -> 10.3 ms (the general kernel of vss.cu -> this one; cutting the last
// round's distributions over radii is 15 % of it); error against 64-bit arithmetic
// 4.0e-6 -> 3.5e-6 to 3.7e-6 of Q.  Bound: shared memory (57 %), the FP32 pipe (48 %)
// and the barriers between passes.  (The factors are real but for Nyquist terms; packing them as
// one complex transform drops those terms, 1e-3 of Q on this mixture.)
#include <algorithm>

#include "common.cuh"
#include "fft_codelets.cuh"
#include "split.cuh"
#include "tcgen05.cuh"

namespace bdgfs {

namespace vssp {
constexpr int N = 24, n = N * N * N, NZ = N * N, NT = 320;
constexpr int RP = N + 1, PX = N * RP;                       // pitches of y and x
constexpr int kTask = 4 * N;                                 // TMEM columns of a task: G^ of both species
constexpr size_t kCube = size_t(N) * PX * sizeof(float4);
constexpr size_t kSmem = kCube + 3 * N * sizeof(float4);
constexpr size_t kF = size_t(N) * NZ * sizeof(float4);       // F of both species
constexpr size_t kSlot = size_t(N) * NZ * sizeof(float4);    // partial G^ of both species
}  // namespace vssp

struct VssPairArgs {
    bdgfs_vss_pair_args g;
    unsigned char* F;                // [CTA] kF
    unsigned char* sums;             // [CTA] kSlot: sum of the radii
    unsigned char* slots;            // [cut distribution][radius] kSlot
    uint32_t* tickets;               // [cut distribution], zeroed
    SplitPlan plan;
};

__device__ __forceinline__ float2 v2(float a, float b) { return make_float2(a, b); }
__device__ __forceinline__ float2 neg2(float2 a) { return make_float2(-a.x, -a.y); }

// The thread's accumulators (ntask pencils in tensor memory) to zero, and out to
// ``to`` [kx][NZ], added to what it holds if ``add``.  Once per radius: calls, so that
// their registers do not count in the slices' loop.
__device__ __noinline__ void vssp_clear(uint32_t tcol, int ntask)
{
    uint32_t zero[16];
#pragma unroll
    for (int k = 0; k < 16; ++k) zero[k] = 0u;
    for (int c = 0; c < ntask * (vssp::kTask / 16); ++c) tc::tmem_st16(tcol + 16 * c, zero);
    tc::tmem_wait_st();
}

__device__ __noinline__ void vssp_flush(uint32_t tcol, int ntask, float4* to, bool add)
{
    using namespace vssp;
    tc::tmem_wait_st();
    for (int r = 0; r < ntask; ++r) {
        for (int cc = 0; cc < N / 8; ++cc) {
            float4* o = to + 8 * cc * NZ + r * NT;
            float4 t[8];                                        // loads before the stores
#pragma unroll
            for (int k = 0; k < 8; ++k) t[k] = add ? __ldcg(o + k * NZ) : make_float4(0.f, 0.f, 0.f, 0.f);
            uint32_t u[16], q[16];
            tc::tmem_ld16_issue(tcol + r * kTask + 16 * cc, u);
            tc::tmem_ld16_issue(tcol + r * kTask + 2 * N + 16 * cc, q);
            tc::tmem_wait();
#pragma unroll
            for (int k = 0; k < 8; ++k)
                __stcg(o + k * NZ, make_float4(__fadd_rn(t[k].x, __uint_as_float(u[2 * k])), __fadd_rn(t[k].y, __uint_as_float(u[2 * k + 1])),
                                               __fadd_rn(t[k].z, __uint_as_float(q[2 * k])), __fadd_rn(t[k].w, __uint_as_float(q[2 * k + 1]))));
        }
    }
}

// The thread's pencils of the Nrho slots at ``from``, added in order into ``to``.  A
// call of its own: inside the last stage its loop cost the slices 110 bytes of
// spills (370 pairs: 10.9 -> 10.5 ms).
__device__ __noinline__ void vssp_merge(const float4* from, float4* to, int Nrho, int ntask)
{
    using namespace vssp;
    for (int r = 0; r < ntask; ++r, from += NT, to += NT) {
        float4 s[N];
#pragma unroll
        for (int k = 0; k < N; ++k) s[k] = __ldcg(from + k * NZ);
#pragma unroll 1
        for (int j = 1; j < Nrho; ++j) {
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const float4 v = __ldcg(from + size_t(j) * N * NZ + k * NZ);
                s[k] = make_float4(__fadd_rn(s[k].x, v.x), __fadd_rn(s[k].y, v.y), __fadd_rn(s[k].z, v.z), __fadd_rn(s[k].w, v.w));
            }
        }
#pragma unroll
        for (int k = 0; k < N; ++k) __stcg(to + k * NZ, s[k]);
    }
}

// NaN in place of what a CTA gives of which a wait ran out
__device__ __noinline__ void vssp_lose(float* p, int n)
{
    for (int i = 0; i < n; ++i) p[i] = __int_as_float(0x7fffffff);
}

__global__ void __launch_bounds__(vssp::NT, 1) vss_pair_kernel(const VssPairArgs a)
{
    using namespace vssp;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ uint32_t s_tmem;
    __shared__ int s_last;
    __shared__ volatile int s_lost;
    __shared__ __align__(8) uint64_t s_free;
    const bdgfs_vss_pair_args& g = a.g;
    float4* W = reinterpret_cast<float4*>(smem);
    float2* T = reinterpret_cast<float2*>(smem);
    float4* E = W + N * PX;                                    // [axis][k]: (E1.re, E2.re, E1.im, E2.im)
    const int tid = threadIdx.x, warp = tid >> 5;
    if (tid < 32) tc::tmem_alloc(&s_tmem, 512);
    if (tid == 0) {
        tc::mbar_init(&s_free, NT);
        s_lost = 0;
    }
    tc::tc_fence_before();
    __syncthreads();
    tc::tc_fence_after();
    // task r of the thread: pencil tid + r * 320; warps 0-7 have two (their
    // TMEM columns 0..191 or 192..383), warps 8 and 9 one (384..479)
    const int ntask = tid + NT < NZ ? 2 : 1;
    const uint32_t tcol = s_tmem + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(2 * kTask * (warp >> 2));

    uint32_t par = 1;
    auto wait_free = [&]() {                                    // bounded; on expiry the CTA gives NaN
        tc::mbar_wait_or_lose(&s_free, par, &s_lost);
        par ^= 1u;
        __syncwarp();
    };
    auto arrive = [&]() { tc::mbar_arrive(&s_free); };
    // cube addresses: pencil t = i * 24 + j of each pass
    auto at_x = [](int t) { return (t / N) * RP + t % N; };            // (y, z): + x * PX
    auto at_y = [](int t) { return (t / N) * PX + t % N; };            // (x, z): + y * RP
    auto at_z = [](int t) { return (t / N) * PX + (t % N) * RP; };     // (x, y): + z
    auto t_row = [](int x, int y) { return 2 * (x * PX + y * RP) + ((3 * x + (y >> 3)) & 1); };  // product: + z
    auto get = [&](int b, int s, float2 (&vr)[N], float2 (&vi)[N]) {
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float4 v = W[b + k * s];
            vr[k] = v2(v.x, v.y);
            vi[k] = v2(v.z, v.w);
        }
    };
    auto put = [&](int b, int s, const float2 (&vr)[N], const float2 (&vi)[N]) {
#pragma unroll
        for (int k = 0; k < N; ++k) W[b + k * s] = make_float4(vr[k].x, vr[k].y, vi[k].x, vi[k].y);
    };
    auto pass_y_inv = [&]() {
#pragma unroll 1
        for (int r = 0; r < ntask; ++r) {
            const int b = at_y(tid + r * NT);
            float2 vr[N], vi[N];
            get(b, RP, vr, vi);
            dft_p2<N, +1>(vr, vi);
            put(b, RP, vr, vi);
        }
    };

    float4* F = reinterpret_cast<float4*>(a.F + size_t(blockIdx.x) * kF);      // [kx][ky*24 + kz]: (F0.re, F1.re, F0.im, F1.im)
    const int Nrho = g.Nrho, M = g.M;
    const float4* phase = static_cast<const float4*>(g.phase);
    const float* bself = static_cast<const float*>(g.bself);
    const float4* bcross = static_cast<const float4*>(g.bcross);
    const float2* c = static_cast<const float2*>(g.c);
    const int64_t nitems = split_items(g.ndof, a.plan);
    for (int64_t item = blockIdx.x; item < nitems; item += gridDim.x) {
        const SplitItem it = split_item(item, a.plan, Nrho);
        const int64_t dof = it.li;
        const int ns = it.ns;
        const float* f0 = static_cast<const float*>(g.f[0]) + dof * n;
        const float* f1 = static_cast<const float*>(g.f[1]) + dof * n;

        // ---- F_p = FFT(f_p) / n, both species ----
        wait_free();
#pragma unroll 1
        for (int r = 0; r < ntask; ++r) {
            const int t = tid + r * NT;
            float2 vr[N], vi[N];
#pragma unroll
            for (int z = 0; z < N; ++z) {
                vr[z] = v2(f0[t * N + z], f1[t * N + z]);
                vi[z] = v2(0.f, 0.f);
            }
            dft_p2<N, -1>(vr, vi);
            put(at_z(t), 1, vr, vi);
        }
        __syncthreads();
#pragma unroll 1
        for (int r = 0; r < ntask; ++r) {
            const int b = at_y(tid + r * NT);
            float2 vr[N], vi[N];
            get(b, RP, vr, vi);
            dft_p2<N, -1>(vr, vi);
            put(b, RP, vr, vi);
        }
        __syncthreads();
#pragma unroll 1
        for (int r = 0; r < ntask; ++r) {
            const int t = tid + r * NT;
            float2 vr[N], vi[N];
            get(at_x(t), PX, vr, vi);
            if (r + 1 == ntask) arrive();
            dft_p2<N, -1>(vr, vi);
            const float sc = 1.f / float(n);
#pragma unroll
            for (int k = 0; k < N; ++k)
                F[k * NZ + t] = make_float4(vr[k].x * sc, vr[k].y * sc, vi[k].x * sc, vi[k].y * sc);
        }

        // ---- slices: radius rho, pair kind (0: species 0 with itself, 1: species 1
        // with itself, 2: unlike), direction s; phase tables kind by kind ----
        // G^ of a radius in tensor memory; at its end to the radius' slot (cut) or onto
        // the sum of the radii
        float4* Gs = ns > 1 ? reinterpret_cast<float4*>(a.slots + size_t(it.cut * Nrho) * kSlot)
                            : reinterpret_cast<float4*>(a.sums + size_t(blockIdx.x) * kSlot);
        const int rho1 = it.b1;
        int rho = it.b0, kind = 0, s = 0;
        vssp_clear(tcol, ntask);
        const int half = M / 2;
        auto table = [&](int q, int k, int d) { return (k < 2 ? (k * Nrho + q) * half : (Nrho + q) * M) + d; };
        if (tid < 3 * N) E[tid] = phase[size_t(table(rho, 0, 0)) * 3 * N + tid];
        __syncthreads();
        while (rho < rho1) {
            const int ti = table(rho, kind, s);
            // the slice after this one
            int nrho = rho, nkind = kind, ndir = s + 1;
            if (ndir == (kind < 2 ? half : M)) {
                ndir = 0;
                if (++nkind == 3) {
                    nkind = 0;
                    ++nrho;
                }
            }
            float4 enext = make_float4(0.f, 0.f, 0.f, 0.f);
            if (tid < 3 * N && nrho < rho1) enext = phase[size_t(table(nrho, nkind, ndir)) * 3 * N + tid];
            // x: phases and inverse transform
#pragma unroll 1
            for (int r = 0; r < ntask; ++r) {
                const int t = tid + r * NT;
                const float4 ey = E[N + t / N], ez = E[2 * N + t % N];
                const float2 yr = v2(ey.x, ey.y), yi = v2(ey.z, ey.w), zr = v2(ez.x, ez.y), zi = v2(ez.z, ez.w);
                const float2 er = __ffma2_rn(neg2(yi), zi, __fmul2_rn(yr, zr));
                const float2 ei = __ffma2_rn(yr, zi, __fmul2_rn(yi, zr));
                const float2 nei = neg2(ei);
                float2 vr[N], vi[N];
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const float4 v = F[k * NZ + t];
                    vr[k] = v2(kind == 1 ? v.y : v.x, kind == 0 ? v.x : v.y);
                    vi[k] = v2(kind == 1 ? v.w : v.z, kind == 0 ? v.z : v.w);
                }
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const float4 x = E[k];
                    const float2 xr = v2(x.x, x.y), xi = v2(x.z, x.w);
                    const float2 cr = __ffma2_rn(xi, nei, __fmul2_rn(xr, er));
                    const float2 ci = __ffma2_rn(xi, er, __fmul2_rn(xr, ei));
                    const float2 re = __ffma2_rn(neg2(ci), vi[k], __fmul2_rn(cr, vr[k]));
                    vi[k] = __ffma2_rn(ci, vr[k], __fmul2_rn(cr, vi[k]));
                    vr[k] = re;
                }
                dft_p2<N, +1>(vr, vi);
                if (r == 0) wait_free();
                put(at_x(t), PX, vr, vi);
            }
            __syncthreads();
            if (tid < 3 * N) E[tid] = enext;                    // read after the next barriers
            pass_y_inv();
            __syncthreads();
            // z: inverse transform, product, forward transform
#pragma unroll 1
            for (int r = 0; r < ntask; ++r) {
                const int t = tid + r * NT;
                cpx<float> X[N];
                {
                    float2 vr[N], vi[N];
                    get(at_z(t), 1, vr, vi);
                    dft_p2<N, +1>(vr, vi);
#pragma unroll
                    for (int z = 0; z < N; ++z)
                        X[z] = {fmaf(vr[z].x, vr[z].y, -vi[z].x * vi[z].y), fmaf(vr[z].x, vi[z].y, vi[z].x * vr[z].y)};
                }
                dft<N, -1>(X);
                const int b = t_row(t / N, t % N);
#pragma unroll
                for (int k = 0; k < N; ++k) T[b + k] = v2(X[k].x, X[k].y);
            }
            __syncthreads();
            // y: forward transform of the product
#pragma unroll 1
            for (int r = 0; r < ntask; ++r) {
                const int t = tid + r * NT, x = t / N, z = t % N;
                cpx<float> X[N];
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const float2 v = T[t_row(x, k) + z];
                    X[k] = {v.x, v.y};
                }
                dft<N, -1>(X);
#pragma unroll
                for (int k = 0; k < N; ++k) T[t_row(x, k) + z] = v2(X[k].x, X[k].y);
            }
            __syncthreads();
            // x: forward transform, weighted into G^
#pragma unroll 1
            for (int r = 0; r < ntask; ++r) {
                const int t = tid + r * NT, y = t / N, z = t % N;
                cpx<float> X[N];
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const float2 v = T[t_row(k, y) + z];
                    X[k] = {v.x, v.y};
                }
                if (r + 1 == ntask) arrive();
                dft<N, -1>(X);
                tc::tmem_wait_st();
                const uint32_t col = tcol + r * kTask;
                if (kind < 2) {
                    const float* w = bself + size_t(ti) * n + t;
#pragma unroll
                    for (int cc = 0; cc < N / 8; ++cc) {
                        float b[8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) b[k] = ldg(w + (8 * cc + k) * NZ);
                        uint32_t u[16];
                        tc::tmem_ld16_issue(col + kind * 2 * N + 16 * cc, u);
                        tc::tmem_wait();
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const cpx<float> x = X[8 * cc + k];
                            u[2 * k] = __float_as_uint(fmaf(b[k], x.x, __uint_as_float(u[2 * k])));
                            u[2 * k + 1] = __float_as_uint(fmaf(b[k], x.y, __uint_as_float(u[2 * k + 1])));
                        }
                        tc::tmem_st16(col + kind * 2 * N + 16 * cc, u);
                    }
                } else {
                    const float4* w = bcross + size_t(ti - Nrho * M) * n + t;
#pragma unroll
                    for (int cc = 0; cc < N / 8; ++cc) {
                        float4 b[8];
#pragma unroll
                        for (int k = 0; k < 8; ++k) b[k] = __ldg(w + (8 * cc + k) * NZ);
                        uint32_t u[16], q[16];
                        tc::tmem_ld16_issue(col + 16 * cc, u);
                        tc::tmem_ld16_issue(col + 2 * N + 16 * cc, q);
                        tc::tmem_wait();
#pragma unroll
                        for (int k = 0; k < 8; ++k) {
                            const cpx<float> x = X[8 * cc + k];
                            const float4 v = b[k];
                            u[2 * k] = __float_as_uint(fmaf(v.x, x.x, fmaf(-v.y, x.y, __uint_as_float(u[2 * k]))));
                            u[2 * k + 1] = __float_as_uint(fmaf(v.x, x.y, fmaf(v.y, x.x, __uint_as_float(u[2 * k + 1]))));
                            q[2 * k] = __float_as_uint(fmaf(v.z, x.x, fmaf(-v.w, x.y, __uint_as_float(q[2 * k]))));
                            q[2 * k + 1] = __float_as_uint(fmaf(v.z, x.y, fmaf(v.w, x.x, __uint_as_float(q[2 * k + 1]))));
                        }
                        tc::tmem_st16(col + 16 * cc, u);
                        tc::tmem_st16(col + 2 * N + 16 * cc, q);
                    }
                }
            }
            if (nrho != rho) {                                  // the radius' last slice
                vssp_flush(tcol, ntask, (ns > 1 ? Gs + size_t(rho) * N * NZ : Gs) + tid, ns == 1 && rho > 0);
                if (nrho < rho1) vssp_clear(tcol, ntask);
            }
            rho = nrho;
            kind = nkind;
            s = ndir;
        }

        if (ns > 1) {
            if (s_lost) vssp_lose(reinterpret_cast<float*>(Gs + size_t(it.b0) * N * NZ + tid), 4);
            __threadfence();
            __syncthreads();
            if (tid == 0) s_last = atomicAdd(a.tickets + it.cut, 1u) == uint32_t(ns - 1);
            __syncthreads();
            if (!s_last) continue;
            __threadfence();
            float4* sum = reinterpret_cast<float4*>(a.sums + size_t(blockIdx.x) * kSlot);
            vssp_merge(Gs + tid, sum + tid, Nrho, ntask);
            Gs = sum;
        }

        // ---- back to velocity space: lane A QG_p, lane B QL_p; Q_p = QG_p - f_p QL_p ----
#pragma unroll 1
        for (int p = 0; p < 2; ++p) {
#pragma unroll 1
            for (int r = 0; r < ntask; ++r) {
                const int t = tid + r * NT;
                float2 vr[N], vi[N];
                const float2* sp = reinterpret_cast<const float2*>(Gs) + 2 * t + p;
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const float2 v = __ldcg(sp + 2 * k * NZ);
                    vr[k].x = v.x;
                    vi[k].x = v.y;
                }
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const float4 v = F[k * NZ + t];
                    const float2 ca = __ldg(c + size_t(2 * p) * n + k * NZ + t);
                    const float2 cb = __ldg(c + size_t(2 * p + 1) * n + k * NZ + t);
                    vr[k].y = ca.x * v.x - ca.y * v.z + cb.x * v.y - cb.y * v.w;
                    vi[k].y = ca.x * v.z + ca.y * v.x + cb.x * v.w + cb.y * v.y;
                }
                dft_p2<N, +1>(vr, vi);
                if (r == 0) wait_free();
                put(at_x(t), PX, vr, vi);
            }
            __syncthreads();
            pass_y_inv();
            __syncthreads();
            const float* fp = p ? f1 : f0;
            float* Q = static_cast<float*>(g.Q[p]) + dof * n;
#pragma unroll 1
            for (int r = 0; r < ntask; ++r) {
                const int t = tid + r * NT;
                float2 vr[N], vi[N];
                get(at_z(t), 1, vr, vi);
                if (r + 1 == ntask) arrive();
                dft_p2<N, +1>(vr, vi);
#pragma unroll
                for (int z = 0; z < N; ++z) Q[t * N + z] = vr[z].x - fp[t * N + z] * vr[z].y;
                if (s_lost) vssp_lose(Q + t * N, N);
            }
        }
    }
    tc::tmem_wait_st();
    tc::tc_fence_before();
    __syncthreads();
    if (tid < 32) {
        tc::tc_fence_after();
        tc::tmem_dealloc(s_tmem, 512);
    }
}

}  // namespace bdgfs

using namespace bdgfs;

// scratch: [tickets, padding][F per CTA][sum per CTA][slots]
static size_t vssp_head(int64_t nslots) { return (size_t(nslots + 1) * sizeof(uint32_t) + 255) / 256 * 256; }

extern "C" int64_t bdgfs_vss_pair_scratch_bytes(int32_t nctas)
{
    if (nctas < 1) return 0;
    // F and the sum per CTA, and seven slots for the radii of cut distributions
    return int64_t(vssp_head(7 * int64_t(nctas)) + size_t(nctas) * (vssp::kF + 8 * vssp::kSlot) + 256);
}

extern "C" int64_t bdgfs_vss_pair_scratch_for(int32_t nctas, int64_t ndof, int32_t Nrho)
{
    if (nctas < 1 || ndof < 1 || Nrho < 1) return 0;
    // CTAs with work, and the slots of the last round's distributions where those of
    // nctas CTAs are enough to cut it
    const int64_t ctas = ndof >= nctas ? nctas : std::min<int64_t>(nctas, ndof * Nrho);
    const int64_t cut = ndof % ctas * Nrho, nslots = cut <= 7 * int64_t(nctas) ? cut : 0;
    return int64_t(vssp_head(nslots) + size_t(ctas) * (vssp::kF + vssp::kSlot) + size_t(nslots) * vssp::kSlot + 256);
}

extern "C" int32_t bdgfs_vss_pair_collide(const bdgfs_vss_pair_args* g, void* scratch, int64_t bytes, void* stream)
{
    using namespace vssp;
    if (!g || !scratch || g->ndof < 0 || g->Nrho < 1 || g->M < 2 || g->M % 2 || !g->phase || !g->bself || !g->bcross ||
        !g->c || !g->f[0] || !g->f[1] || !g->Q[0] || !g->Q[1])
        return BDGFS_EINVAL;
    if (g->Nv != N) return BDGFS_EUNSUPPORTED;
    if (g->ndof == 0) return BDGFS_OK;
    int dev = 0, nsm = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return BDGFS_ECUDA;
    if (cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, dev) != cudaSuccess) return BDGFS_ECUDA;
    // CTAs and slots that fit
    const uintptr_t base = (reinterpret_cast<uintptr_t>(scratch) + 255) & ~uintptr_t(255);
    const int64_t room = bytes - int64_t(base - reinterpret_cast<uintptr_t>(scratch));
    const int64_t work = g->ndof >= nsm ? nsm : std::min<int64_t>(nsm, g->ndof * g->Nrho);
    int64_t nctas = std::min<int64_t>(work, (room - int64_t(vssp_head(0))) / int64_t(kF + kSlot));
    if (nctas < 1) return BDGFS_ESCRATCH;
    int64_t nslots = 0;
    while (int64_t(vssp_head(nslots + 1) + size_t(nctas) * (kF + kSlot) + size_t(nslots + 1) * kSlot) <= room &&
           nslots < 7 * int64_t(nsm))
        ++nslots;
    VssPairArgs a{};
    a.g = *g;
    a.plan = split_plan(g->ndof, nslots, g->Nrho, int(nctas), 0.3f, 0.4f);
    a.tickets = reinterpret_cast<uint32_t*>(base);
    a.F = reinterpret_cast<unsigned char*>(base + vssp_head(nslots));
    a.sums = a.F + size_t(nctas) * kF;
    a.slots = a.sums + size_t(nctas) * kSlot;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const size_t cut = size_t(g->ndof - a.plan.whole);
    if (cut > 0 && cudaMemsetAsync(a.tickets, 0, sizeof(uint32_t) * cut, st) != cudaSuccess) return BDGFS_ECUDA;
    if (const int rc = smem_optin(reinterpret_cast<const void*>(vss_pair_kernel), kSmem)) return rc;
    nctas = std::min(nctas, split_items(g->ndof, a.plan));
    vss_pair_kernel<<<unsigned(nctas), NT, kSmem, st>>>(a);
    return cuda_status(cudaGetLastError());
}
