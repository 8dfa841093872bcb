// Collision operator with the exact Nyquist term on small grids (Nv = 8, 12,
// 16; both precisions): included by vhs_collide.cu, whose header states the
// algorithm's quantities.
//
// BDGFS_EXACT subtracts Re(w_s^2), w_s = IFFT(i m_s F), from each S_p term.  m_s
// vanishes off the Nyquist planes, so w_s is a sum of three 2-D transforms,
//   w_s = (-1)^x X(y, z) + (-1)^y Y(x, z) + (-1)^z Z(x, y),
// X from the plane kx = N/2, Y from ky = N/2 without kx = N/2, Z from kz = N/2
// without the other two: 6 N pencils a direction instead of the 3 N^2 of a second
// 3-D transform.  They are done for up to kQB directions at a time (6 N kQB
// pencils keep every warp busy) before those directions' transforms, and enter
// where S_p is updated.
//
// The multiplier of any pencil is m = al Ez.x + be Ez.y (be2 at kz = N/2) with
// per-pencil al, be, be2, so Nyquist pencils take no branch of their own.
//
// One CTA of N^2 threads per distribution, a pencil per thread; short lists and the
// last round of a long one are cut over radii (split.cuh).  Measured on one B200,
// 16^3, Nrho = 8, 6 directions, exact term, 144 distributions in FP64: 0.297 ->
// 0.188 ms (the general variant with its second transform -> this one; error
// against 64 bits unchanged); without the term 2048 in FP32: 2.21 -> 1.24 ms.
// Bound in FP64: shared memory (62 %, and its latency at eight warps an SM) and
// the FP64 pipe (46 %).
#pragma once
#include "split.cuh"

namespace bdgfs {

// products and sums that are not contracted: cut and whole distributions get the
// same bits
__device__ __forceinline__ float add_rn(float a, float b) { return __fadd_rn(a, b); }
__device__ __forceinline__ double add_rn(double a, double b) { return __dadd_rn(a, b); }
__device__ __forceinline__ float mul_rn(float a, float b) { return __fmul_rn(a, b); }
__device__ __forceinline__ double mul_rn(double a, double b) { return __dmul_rn(a, b); }

template <typename T, int N>
struct Exact {
    static constexpr int H = N / 2, NH = H + 1, NP = N * N, NT = (NP + 31) / 32 * 32;
    static constexpr int WS = N + 1;
    static constexpr int kQB = 6;                              // directions per plane batch
    static constexpr size_t kPlane = size_t(N) * WS;
    static size_t smem_bytes(int M)
    {
        const int qb = M < kQB ? M : kQB;
        size_t b = (size_t(N) * N * WS + size_t(NH) * N * WS + size_t(M) * 3 * N + size_t(qb) * 3 * kPlane) * sizeof(cpx<T>);
        return b + 10 * (NT / 32) * sizeof(double) + 16;
    }
    static constexpr size_t slot_bytes() { return (size_t(N) * NH * N * sizeof(cpx<T>) + 255) / 256 * 256; }
    // per SM: a slot for each of up to four CTAs, and eight for the radii of cut
    // distributions
    static constexpr int kCtas = 4, kCut = 8;
    static size_t scratch_bytes() { return (kCtas + kCut) * (slot_bytes() + 256); }
};

struct ExactArgs {
    bdgfs_vhs_grid g;
    bdgfs_vhs_batch batches[4];
    int32_t nbatch, flags;
    unsigned char* slots;
    uint32_t* tickets;
    SplitArgs split;                // slots: radii of cut distributions, after one per CTA
    unsigned long long* counter;
};

// m(kz) = a Ez.x + b Ez.y, b2 for b at kz = N/2: multiplier (tr = 0) or Nyquist
// term (tr = 1) of pencil (kx, ky)
template <typename T, int N>
__device__ __forceinline__ void exact_coef(const cpx<T>* ep, int kx, int ky, int tr, T& a, T& b, T& b2)
{
    const cpx<T> Ex = ep[kx], Ey = ep[N + ky];
    const cpx<T> P = cmul(Ex, Ey);
    const cpx<T> Pb = cmul(kx == N / 2 ? Ex : conjc(Ex), ky == N / 2 ? Ey : conjc(Ey));
    const T h = T(0.5);
    if (tr == 0) {
        a = h * ((P.x + P.y) + (Pb.x - Pb.y));
        b = h * ((P.x - P.y) + (Pb.x + Pb.y));
        b2 = h * ((P.x - P.y) - (Pb.x + Pb.y));
    } else {
        a = h * ((P.y - P.x) + (Pb.x + Pb.y));
        b = h * ((P.x + P.y) + (Pb.y - Pb.x));
        b2 = h * ((P.x + P.y) + (Pb.x - Pb.y));
    }
}

template <typename T, int N>
__global__ void __launch_bounds__(Exact<T, N>::NT) vhs_exact_kernel(const ExactArgs a)
{
    using X = Exact<T, N>;
    constexpr int H = X::H, NH = X::NH, NP = X::NP, NT = X::NT, WS = X::WS, n = N * N * N;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int64_t s_item;
    __shared__ int64_t s_start[5];
    __shared__ SplitPlan s_plan;
    __shared__ int s_last;
    const bdgfs_vhs_grid& g = a.g;
    const int tid = threadIdx.x, M = g.M, Nrho = g.Nrho;
    cpx<T>* W = reinterpret_cast<cpx<T>*>(smem);
    cpx<T>* Fh = W + N * N * WS;
    cpx<T>* ph = Fh + NH * N * WS;
    cpx<T>* pln = ph + M * 3 * N;                              // [qi][plane][i][j]
    double* red = reinterpret_cast<double*>(
        (reinterpret_cast<uintptr_t>(pln + size_t(min(M, X::kQB)) * 3 * X::kPlane) + 15) & ~uintptr_t(15));
    const cpx<T>* phase = static_cast<const cpx<T>*>(g.phase);
    const T* gw = static_cast<const T*>(g.gw);
    const T* bb2 = static_cast<const T*>(g.bb2);
    const int project = a.flags & BDGFS_PROJECT;
    const bool exact = a.flags & BDGFS_EXACT;
    if (tid == 0) {
        s_start[0] = 0;
        for (int b = 0; b < a.nbatch; ++b) {
            int64_t c = a.batches[b].ndof;
            if (a.batches[b].count) {
                const int64_t d = *a.batches[b].count;
                c = d < 0 ? 0 : (d < c ? d : c);
            }
            s_start[b + 1] = s_start[b] + c;
        }
        s_plan = split_plan(a.split, s_start[a.nbatch], Nrho);
    }
    __syncthreads();
    // pencil of every pass; threads beyond N^2 (Nv = 12) take no part
    const bool on = tid < NP;
    const int pa = on ? tid / N : 0, pb = on ? tid % N : 0;
    auto w = [&](int i, int j, int k) -> cpx<T>& { return W[(i * N + j) * WS + k]; };
    // F(kx, ky, kz) from its half kx <= N/2
    auto Fat = [&](int kx, int ky, int kz) {
        if (kx < NH) return Fh[(kx * N + ky) * WS + kz];
        return conjc(Fh[((N - kx) * N + (N - ky) % N) * WS + (N - kz) % N]);
    };

    const int64_t total = s_start[a.nbatch];
    const SplitPlan plan = s_plan;
    const int64_t nitems = split_items(total, plan);
    for (;;) {
        if (tid == 0) s_item = int64_t(atomicAdd(a.counter, 1ull));
        __syncthreads();
        const int64_t item = s_item;
        __syncthreads();
        if (item >= nitems) break;
        const SplitItem it = split_item(item, plan, Nrho);
        const int64_t li = it.li;
        const int ns = it.ns;
        int b = 0;
        while (li >= s_start[b + 1]) ++b;
        const bdgfs_vhs_batch& bt = a.batches[b];
        const int64_t pos = li - s_start[b];
        const int64_t dof = bt.index ? int64_t(bt.index[pos]) : pos;
        if (dof < 0 || dof >= bt.ndof) continue;               // malformed index list: skip
        const T* f = static_cast<const T*>(bt.f) + dof * n;

        cpx<T> v[N];
        // ---- Fh = FFT(f) / n, kx <= N/2 ----
        if (on) {
#pragma unroll
            for (int x = 0; x < N; ++x) v[x] = {f[(x * N + pa) * N + pb], T(0)};
            dft<N, -1>(v);
#pragma unroll
            for (int kx = 0; kx < NH; ++kx) w(kx, pa, pb) = v[kx];
        }
        // forward y and z passes of the half spectrum in W
        auto forward_yz = [&]() {
            __syncthreads();
            if (tid < NH * N) {
#pragma unroll
                for (int j = 0; j < N; ++j) v[j] = w(pa, j, pb);
                dft<N, -1>(v);
#pragma unroll
                for (int j = 0; j < N; ++j) w(pa, j, pb) = v[j];
            }
            __syncthreads();
            if (tid < NH * N) {
#pragma unroll
                for (int k = 0; k < N; ++k) v[k] = w(pa, pb, k);
                dft<N, -1>(v);
            }
        };
        forward_yz();
        if (tid < NH * N) {
            const T sc = T(1) / T(n);
#pragma unroll
            for (int k = 0; k < N; ++k) Fh[(pa * N + pb) * WS + k] = {v[k].x * sc, v[k].y * sc};
        }

        // G^ [kz][kx][ky]: the sum so far, or one slot per radius (cut)
        auto slot_at = [&](int64_t i) { return reinterpret_cast<cpx<T>*>(a.slots + size_t(i) * X::slot_bytes()); };
        cpx<T>* G = slot_at(blockIdx.x);
        for (int p = it.b0; p < it.b1; ++p) {
            for (int e = tid; e < M * 3 * N; e += NT) ph[e] = phase[size_t(p) * M * 3 * N + e];
            T S[N];
#pragma unroll
            for (int x = 0; x < N; ++x) S[x] = T(0);
            __syncthreads();                                   // phases and Fh in place, W free
            for (int q0 = 0; q0 < M; q0 += X::kQB) {
                const int nq = min(M - q0, X::kQB);
                if (exact) {
                    // planes: first axis (z of X and Y, y of Z), then the other, in place
#pragma unroll 1
                    for (int t = tid; t < nq * 3 * N; t += NT) {
                        const int i = t % N, pl = (t / N) % 3, qi = t / (3 * N);
                        const cpx<T>* ep = ph + (q0 + qi) * 3 * N;
                        if (pl < 2) {
                            const int kx = pl ? i : H, ky = pl ? H : i;
                            T ca, cb, cb2;
                            exact_coef<T, N>(ep, kx, ky, 1, ca, cb, cb2);
                            if (pl && i == H) ca = cb = cb2 = T(0);     // in X already
#pragma unroll
                            for (int kz = 0; kz < N; ++kz) {
                                const cpx<T> Ez = ep[2 * N + kz], F = Fat(kx, ky, kz);
                                const T m = ca * Ez.x + (kz == H ? cb2 : cb) * Ez.y;
                                v[kz] = {-m * F.y, m * F.x};
                            }
                        } else {
                            // kx, ky off their Nyquist planes: m_s = (Re + Im)(Ex Ey) Im Ez(N/2)
                            const cpx<T> Ex = ep[i];
                            const T s = i == H ? T(0) : ep[2 * N + H].y;
#pragma unroll
                            for (int ky = 0; ky < N; ++ky) {
                                const cpx<T> P = cmul(Ex, ep[N + ky]), F = Fat(i, ky, H);
                                const T m = ky == H ? T(0) : (P.x + P.y) * s;
                                v[ky] = {-m * F.y, m * F.x};
                            }
                        }
                        dft<N, +1>(v);
                        cpx<T>* o = pln + (qi * 3 + pl) * X::kPlane + i * WS;
#pragma unroll
                        for (int k = 0; k < N; ++k) o[k] = v[k];
                    }
                    __syncthreads();
#pragma unroll 1
                    for (int t = tid; t < nq * 3 * N; t += NT) {
                        cpx<T>* o = pln + (t / N) * X::kPlane + t % N;
#pragma unroll
                        for (int k = 0; k < N; ++k) v[k] = o[k * WS];
                        dft<N, +1>(v);
#pragma unroll
                        for (int k = 0; k < N; ++k) o[k * WS] = v[k];
                    }
                    // (read after the transform's barriers)
                }
#pragma unroll 1
                for (int qi = 0; qi < nq; ++qi) {
                    const cpx<T>* ep = ph + (q0 + qi) * 3 * N;
                    if (on) {                                  // z: spectrum and inverse transform
                        T ca, cb, cb2;
                        exact_coef<T, N>(ep, pa, pb, 0, ca, cb, cb2);
                        const bool direct = pa < NH;
                        const cpx<T>* fp = Fh + (direct ? pa * N + pb : (N - pa) * N + (N - pb) % N) * WS;
#pragma unroll
                        for (int kz = 0; kz < N; ++kz) {
                            const cpx<T> Ez = ep[2 * N + kz];
                            const cpx<T> F = fp[direct ? kz : (N - kz) % N];
                            const T m = ca * Ez.x + (kz == H ? cb2 : cb) * Ez.y;
                            v[kz] = {m * F.x, direct ? m * F.y : -m * F.y};
                        }
                        dft<N, +1>(v);
#pragma unroll
                        for (int z = 0; z < N; ++z) w(pa, pb, z) = v[z];
                    }
                    __syncthreads();
                    if (on) {                                  // y
#pragma unroll
                        for (int j = 0; j < N; ++j) v[j] = w(pa, j, pb);
                        dft<N, +1>(v);
#pragma unroll
                        for (int j = 0; j < N; ++j) w(pa, j, pb) = v[j];
                    }
                    __syncthreads();
                    if (on) {                                  // x, S_p += Re(w^2) - Re(w_s^2)
#pragma unroll
                        for (int i = 0; i < N; ++i) v[i] = w(i, pa, pb);
                    }
                    __syncthreads();                           // W free for the next transform
                    if (on) {
                        dft<N, +1>(v);
                        if (exact) {
                            const cpx<T>* o = pln + qi * 3 * X::kPlane;
                            const cpx<T> px = o[pa * WS + pb];
                            const T sy = (pa & 1) ? T(-1) : T(1), sz = (pb & 1) ? T(-1) : T(1);
#pragma unroll
                            for (int x = 0; x < N; ++x) {
                                const cpx<T> py = o[X::kPlane + x * WS + pb], pz = o[2 * X::kPlane + x * WS + pa];
                                const T re = (x & 1 ? -px.x : px.x) + sy * py.x + sz * pz.x;
                                const T im = (x & 1 ? -px.y : px.y) + sy * py.y + sz * pz.y;
                                S[x] += (v[x].x + v[x].y) * (v[x].x - v[x].y) - (re + im) * (re - im);
                            }
                        } else {
#pragma unroll
                            for (int x = 0; x < N; ++x) S[x] += (v[x].x + v[x].y) * (v[x].x - v[x].y);
                        }
                    }
                }
                if (exact && q0 + nq < M) __syncthreads();     // planes are read out
            }
            // ---- G^ += gw_p FFT(S_p) (kx <= N/2) ----
            if (on) {
#pragma unroll
                for (int x = 0; x < N; ++x) v[x] = {S[x], T(0)};
                dft<N, -1>(v);
#pragma unroll
                for (int kx = 0; kx < NH; ++kx) w(kx, pa, pb) = v[kx];
            }
            forward_yz();
            if (tid < NH * N) {
                const T* gwp = gw + size_t(p) * N * NH * N + tid;
                cpx<T>* to = (ns > 1 ? slot_at(a.split.nctas + it.cut * Nrho + p) : G) + tid;
                const bool acc = ns == 1 && p > 0;
#pragma unroll
                for (int kz = 0; kz < N; ++kz) {
                    const T wt = ldg(gwp + kz * NH * N);
                    const cpx<T> o = acc ? to[kz * NH * N] : cpx<T>{T(0), T(0)};
                    to[kz * NH * N] = {add_rn(o.x, mul_rn(wt, v[kz].x)), add_rn(o.y, mul_rn(wt, v[kz].y))};
                }
            }
            // (the next radius' staging is followed by a barrier)
        }
        if (ns > 1) {
            // the part that arrives last adds the radii in order and finishes the
            // distribution
            __threadfence();
            __syncthreads();
            if (tid == 0) s_last = atomicAdd(a.tickets + it.cut, 1u) == uint32_t(ns - 1);
            __syncthreads();
            if (!s_last) continue;
            __threadfence();
            if (tid < NH * N) {
                cpx<T> s[N];
#pragma unroll
                for (int kz = 0; kz < N; ++kz) s[kz] = {T(0), T(0)};
#pragma unroll 1
                for (int j = 0; j < Nrho; ++j) {
                    const T* src = reinterpret_cast<const T*>(slot_at(a.split.nctas + it.cut * Nrho + j) + tid);
#pragma unroll
                    for (int kz = 0; kz < N; ++kz) {
                        s[kz].x = add_rn(s[kz].x, __ldcg(src + 2 * kz * NH * N));
                        s[kz].y = add_rn(s[kz].y, __ldcg(src + 2 * kz * NH * N + 1));
                    }
                }
#pragma unroll
                for (int kz = 0; kz < N; ++kz) G[kz * NH * N + tid] = s[kz];
            }
        }
        __syncthreads();

        // ---- QG + i fC = IFFT(G^ + i bb2 Fh) ----
        if (on) {
            const bool direct = pa < NH;
            const int pkx = direct ? pa : N - pa, pky = direct ? pb : (N - pb) % N;
#pragma unroll
            for (int kz = 0; kz < N; ++kz) {
                const int pkz = direct ? kz : (N - kz) % N;
                cpx<T> Gv = G[(pkz * NH + pkx) * N + pky];
                cpx<T> F = Fh[(pkx * N + pky) * WS + pkz];
                if (!direct) { Gv.y = -Gv.y; F.y = -F.y; }
                const T bw = ldg(bb2 + (kz * N + pa) * N + pb);
                v[kz] = {Gv.x - bw * F.y, Gv.y + bw * F.x};
            }
            dft<N, +1>(v);
#pragma unroll
            for (int z = 0; z < N; ++z) w(pa, pb, z) = v[z];
        }
        __syncthreads();
        if (on) {
#pragma unroll
            for (int j = 0; j < N; ++j) v[j] = w(pa, j, pb);
            dft<N, +1>(v);
#pragma unroll
            for (int j = 0; j < N; ++j) w(pa, j, pb) = v[j];
        }
        __syncthreads();
        const T prefac = T(g.prefac);
        double* mom = bt.moments ? bt.moments + dof * 10 : nullptr;
        const bool need_m = project || mom;
        double m[5] = {0, 0, 0, 0, 0};
        T q[N];
        const double cy = g.c0[pa], cz = g.c0[pb];
        if (on) {
#pragma unroll
            for (int i = 0; i < N; ++i) v[i] = w(i, pa, pb);
            dft<N, +1>(v);
            double q0 = 0.0, q1 = 0.0, q2 = 0.0;
#pragma unroll
            for (int x = 0; x < N; ++x) {
                q[x] = prefac * (v[x].x - f[(x * N + pa) * N + pb] * v[x].y);
                if (need_m) {
                    const double cx = g.c0[x], d = double(q[x]);
                    q0 += d;
                    q1 += cx * d;
                    q2 += cx * cx * d;
                }
            }
            m[0] = q0;
            m[1] = q1;
            m[2] = cy * q0;
            m[3] = cz * q0;
            m[4] = q2 + (cy * cy + cz * cz) * q0;
        }
        double lam[5] = {0, 0, 0, 0, 0};
        if (need_m) block_sum<5>(m, red);
        if (project) {
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                double s = 0.0;
#pragma unroll
                for (int j = 0; j < 5; ++j) s += g.ginv[i * 5 + j] * m[j];
                lam[i] = s;
            }
        }
        T* Q = static_cast<T*>(bt.Q) + dof * n;
        double m2[5] = {0, 0, 0, 0, 0};
        if (on) {
            const double base = lam[0] + lam[2] * cy + lam[3] * cz + lam[4] * (cy * cy + cz * cz);
            double q0 = 0.0, q1 = 0.0, q2 = 0.0;
#pragma unroll
            for (int x = 0; x < N; ++x) {
                if (project) {
                    const double cx = g.c0[x];
                    const double qc = double(q[x]) - (base + (lam[1] + lam[4] * cx) * cx);
                    q[x] = T(qc);
                    q0 += qc;
                    q1 += cx * qc;
                    q2 += cx * cx * qc;
                }
                __stcs(Q + (x * N + pa) * N + pb, q[x]);
            }
            m2[0] = q0;
            m2[1] = q1;
            m2[2] = cy * q0;
            m2[3] = cz * q0;
            m2[4] = q2 + (cy * cy + cz * cz) * q0;
        }
        if (mom) {
            if (project) block_sum<5>(m2, red);
            if (tid == 0) {
                for (int j = 0; j < 5; ++j) {
                    mom[j] = m[j] * g.cw;
                    mom[5 + j] = project ? m2[j] * g.cw : m[j] * g.cw;
                }
            }
        }
        __syncthreads();                                       // W is read out
    }
}

}  // namespace bdgfs
