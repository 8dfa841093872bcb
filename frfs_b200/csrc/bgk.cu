// BGK relaxation and the ARS IMEX stage update of the 'adgfs' system.
//
// Reference: ADGFSBGKDirectGLLScatteringModel (frfs/solvers/adgfs/
// scattering.py), kernels cmaxwellian / updateMom{q}_ARS
// (kernels/scattering/bgk-direct-gll.mako:4-113) and
// updateDistribution{q}_ARS (linear-common-direct-gll.mako:90-145), driven
// by ARSabcAstdStepper.step (frfs/integrators/std/steppers.py:531-585).
//
// One CTA per distribution.  The reference computes the moments with a
// cuBLAS product against [1, c, |c|^2] cw, stores every stage Maxwellian in
// a full-size bank and updates f in separate launches; here one launch per
// stage reduces the moments (FP64), forms the stage moments and updates f,
// with each Maxwellian built on the fly from separable exponential tables
// (3 Nv exponentials per Maxwellian instead of Nv^3).
//
// ES-BGK ('esbgk-direct-gll': ADGFSESBGKDirectGLLScatteringModel, kernels
// momentNorm / cmaxwellian / updateMom{q}_ARS of esbgk-direct-gll.mako)
// uses 11 moment rows (the five conserved ones and the six raw second
// moments cx^2, cy^2, cz^2, cx cy, cy cz, cz cx) and relaxes to the
// anisotropic Gaussian of the ES tensor; the Gaussian is not separable and
// is evaluated per velocity.
#include "common.cuh"
#include "rows.cuh"

namespace bdgfs {

constexpr double kPi = 3.141592653589793;

// temperature and density of a moment row
__device__ __forceinline__ void row_state(const double (&U)[5], double& rho, double& ux, double& uy, double& uz,
                                          double& T)
{
    rho = U[0];
    ux = U[1] / U[0];
    uy = U[2] / U[0];
    uz = U[3] / U[0];
    T = (U[4] - (U[1] * U[1] + U[2] * U[2] + U[3] * U[3]) / U[0]) / (1.5 * U[0]);
}

// ES Gaussian of an 11-moment row: G(c) = g[0] exp(-q(c - u)), u = g[1..3],
// q(d) = g[4] dx^2 + g[5] dy^2 + g[6] dz^2 + g[7] dx dy + g[8] dy dz + g[9] dz dx
// (the inverse of T_ij = T/Pr delta_ij + 2 (1 - 1/Pr)(P_ij/rho - u_i u_j)).
__device__ __forceinline__ void es_params(const double* U, double Pr, double (&g)[10])
{
    const double rho = U[0], ux = U[1] / rho, uy = U[2] / rho, uz = U[3] / rho;
    const double T = (U[4] - rho * (ux * ux + uy * uy + uz * uz)) / (1.5 * rho);
    const double k = 2.0 * (1.0 - 1.0 / Pr);
    const double txx = T / Pr + k * (U[5] / rho - ux * ux);
    const double tyy = T / Pr + k * (U[6] / rho - uy * uy);
    const double tzz = T / Pr + k * (U[7] / rho - uz * uz);
    const double txy = k * (U[8] / rho - ux * uy);
    const double tyz = k * (U[9] / rho - uy * uz);
    const double tzx = k * (U[10] / rho - uz * ux);
    const double det = txx * (tyy * tzz - tyz * tyz) - txy * (txy * tzz - tyz * tzx)
                       + tzx * (txy * tyz - tyy * tzx);
    const double id = 1.0 / det;
    g[0] = rho / (kPi * sqrt(kPi) * sqrt(det));
    g[1] = ux;
    g[2] = uy;
    g[3] = uz;
    g[4] = (tyy * tzz - tyz * tyz) * id;
    g[5] = (txx * tzz - tzx * tzx) * id;
    g[6] = (txx * tyy - txy * txy) * id;
    g[7] = 2.0 * (tyz * tzx - tzz * txy) * id;
    g[8] = 2.0 * (txy * tzx - txx * tyz) * id;
    g[9] = 2.0 * (txy * tyz - tzx * tyy) * id;
}

__device__ __forceinline__ double es_eval(const double* g, double cx, double cy, double cz)
{
    const double dx = cx - g[1], dy = cy - g[2], dz = cz - g[3];
    const double q = g[4] * dx * dx + g[5] * dy * dy + g[6] * dz * dz + g[7] * dx * dy + g[8] * dy * dz
                     + g[9] * dz * dx;
    return g[0] * exp(-q);
}

// Shakov target of a 14-moment row: S(c) = M(c) (1 + (k q . d)(2 |d|^2 / T - 5)),
// d = c - u, k = 2 (1 - Pr) / (5 rho T^2), q the heat flux
// q_i = Q_i - 2 P_ij u_j + rho u_i |u|^2 - 1.5 rho T u_i; s = {u, 1/T, k q}
__device__ __forceinline__ void shakov_params(const double* U, double Pr, double (&s)[7])
{
    const double rho = U[0], ux = U[1] / rho, uy = U[2] / rho, uz = U[3] / rho;
    const double u2 = ux * ux + uy * uy + uz * uz;
    const double T = (U[4] - rho * u2) / (1.5 * rho);
    const double qx = U[11] - 2.0 * (U[5] * ux + U[8] * uy + U[10] * uz) + rho * ux * u2 - 1.5 * rho * T * ux;
    const double qy = U[12] - 2.0 * (U[8] * ux + U[6] * uy + U[9] * uz) + rho * uy * u2 - 1.5 * rho * T * uy;
    const double qz = U[13] - 2.0 * (U[10] * ux + U[9] * uy + U[7] * uz) + rho * uz * u2 - 1.5 * rho * T * uz;
    const double k = 2.0 * (1.0 - Pr) / (5.0 * rho * T * T);
    s[0] = ux;
    s[1] = uy;
    s[2] = uz;
    s[3] = 1.0 / T;
    s[4] = k * qx;
    s[5] = k * qy;
    s[6] = k * qz;
}

// the Shakov factor 1 + (k q . d)(2 |d|^2 / T - 5) at velocity c
__device__ __forceinline__ double shakov_factor(const double* s, double cx, double cy, double cz)
{
    const double dx = cx - s[0], dy = cy - s[1], dz = cz - s[2];
    return 1.0 + (s[4] * dx + s[5] * dy + s[6] * dz) * (2.0 * (dx * dx + dy * dy + dz * dz) * s[3] - 5.0);
}

template <typename T, int VEC>
__global__ void __launch_bounds__(256) shakov_target_kernel(const double* __restrict__ U, int Nv,
                                                            const double* c0, double Pr, T* __restrict__ S)
{
    __shared__ double cs[kMaxNv];
    __shared__ double ex[3][kMaxNv];
    const int64_t dof = blockIdx.x;
    const int n = Nv * Nv * Nv;
    const double* u = U + dof * 14;
    double sp[7];
    shakov_params(u, Pr, sp);
    const double am = u[0] / pow(kPi / sp[3], 1.5);
    for (int i = threadIdx.x; i < 3 * Nv; i += blockDim.x) {
        const int d = i / Nv, k = i - d * Nv;
        if (d == 0) cs[k] = c0[k];
        const double c = c0[k] - sp[d];
        ex[d][k] = exp(-c * c * sp[3]);
    }
    __syncthreads();
    T* row = S + dof * int64_t(n);
    for (int v = threadIdx.x * VEC; v < n; v += blockDim.x * VEC) {
        uint32_t ix, iy, iz;
        vsplit(uint32_t(v), uint32_t(Nv), ix, iy, iz);
        Chunk<T, VEC> c;
#pragma unroll
        for (int j = 0; j < VEC; ++j)
            c.v[j] = T(am * ex[0][ix] * ex[1][iy] * ex[2][iz + j] * shakov_factor(sp, cs[ix], cs[iy], cs[iz + j]));
        c.store(row + v);
    }
}

template <typename T, int VEC>
__global__ void __launch_bounds__(256) esbgk_gaussian_kernel(const double* __restrict__ U, int Nv,
                                                             const double* c0, double Pr, T* __restrict__ M)
{
    __shared__ double cs[kMaxNv];
    const int64_t dof = blockIdx.x;
    const int n = Nv * Nv * Nv;
    for (int i = threadIdx.x; i < Nv; i += blockDim.x) cs[i] = c0[i];
    double g[10];
    es_params(U + dof * 11, Pr, g);
    __syncthreads();
    T* row = M + dof * int64_t(n);
    for (int v = threadIdx.x * VEC; v < n; v += blockDim.x * VEC) {
        uint32_t ix, iy, iz;
        vsplit(uint32_t(v), uint32_t(Nv), ix, iy, iz);
        Chunk<T, VEC> c;
#pragma unroll
        for (int j = 0; j < VEC; ++j) c.v[j] = T(es_eval(g, cs[ix], cs[iy], cs[iz + j]));
        c.store(row + v);
    }
}

template <typename T, int VEC>
__global__ void __launch_bounds__(256) bgk_maxwellian_kernel(const double* __restrict__ U, int Nv,
                                                             const double* c0, T* __restrict__ M)
{
    __shared__ double ex[3][kMaxNv];
    const int64_t dof = blockIdx.x;
    const int n = Nv * Nv * Nv;
    double u[5];
#pragma unroll
    for (int i = 0; i < 5; ++i) u[i] = U[dof * 5 + i];
    double rho, ux, uy, uz, Tt;
    row_state(u, rho, ux, uy, uz, Tt);
    const double a = rho / pow(kPi * Tt, 1.5), it = 1.0 / Tt;
    for (int i = threadIdx.x; i < 3 * Nv; i += blockDim.x) {
        const int d = i / Nv, j = i - d * Nv;
        const double c = c0[j] - (d == 0 ? ux : d == 1 ? uy : uz);
        ex[d][j] = exp(-c * c * it);
    }
    __syncthreads();
    T* row = M + dof * int64_t(n);
    for (int v = threadIdx.x * VEC; v < n; v += blockDim.x * VEC) {
        uint32_t ix, iy, iz;
        vsplit(uint32_t(v), uint32_t(Nv), ix, iy, iz);
        const double axy = a * ex[0][ix] * ex[1][iy];
        Chunk<T, VEC> c;
#pragma unroll
        for (int j = 0; j < VEC; ++j) c.v[j] = T(axy * ex[2][iz + j]);
        c.store(row + v);
    }
}

// second moments of the Maxwellian of a moment row: rho T/2 + rho u_i^2, rho u_i u_j
__device__ __forceinline__ void maxwell_second(const double* u, double (&t)[6])
{
    double rho, ux, uy, uz, Tt;
    double u5[5] = {u[0], u[1], u[2], u[3], u[4]};
    row_state(u5, rho, ux, uy, uz, Tt);
    t[0] = 0.5 * rho * Tt + rho * ux * ux;
    t[1] = 0.5 * rho * Tt + rho * uy * uy;
    t[2] = 0.5 * rho * Tt + rho * uz * uz;
    t[3] = rho * ux * uy;
    t[4] = rho * uy * uz;
    t[5] = rho * uz * ux;
}

// explicit heat-flux relaxation target of a 14-moment row (Shakov):
// Q(M)_i + (1 - Pr)(q_i - Q_i), Q(M)_i = rho u_i |u|^2 + 2.5 rho T u_i,
// q_i - Q_i = -2 P_ij u_j + rho u_i |u|^2 - 1.5 rho T u_i
__device__ __forceinline__ void shakov_heat(const double* u, double Pr, double (&h)[3])
{
    double rho, ux, uy, uz, Tt;
    double u5[5] = {u[0], u[1], u[2], u[3], u[4]};
    row_state(u5, rho, ux, uy, uz, Tt);
    const double u2 = ux * ux + uy * uy + uz * uz;
    const double v[3] = {ux, uy, uz};
    const double Pu[3] = {u[5] * ux + u[8] * uy + u[10] * uz, u[8] * ux + u[6] * uy + u[9] * uz,
                          u[10] * ux + u[9] * uy + u[7] * uz};
#pragma unroll
    for (int i = 0; i < 3; ++i)
        h[i] = rho * v[i] * u2 + 2.5 * rho * Tt * v[i]
               + (1.0 - Pr) * (-2.0 * Pu[i] + rho * v[i] * u2 - 1.5 * rho * Tt * v[i]);
}

// partial sums that a row's moments are made of, with 256 or 512 threads: a row gives
// the same bits alone and among thousands (512 slots, walked twice by 256 threads:
// ARS-222 step of 2048 rows of 24^3 418 us; 256 slots: 380 us)
constexpr int kRowSlots = 256, kRowWarps = kRowSlots / 32;

// Moments of up to two rows; sums of row r in ms[r] (warp 0 writes them: read after
// the barrier).  256 threads walk both rows at once (both rows' loads are in flight
// together); of 512, each half walks one row: a BDF-2 Shakov step of 315 rows 82 -> 74
// us against every thread on both rows.
template <typename T, int VEC, int NA>
__device__ __forceinline__ void two_row_moments(const T* __restrict__ r0, const T* __restrict__ r1, int n, int Nv,
                                                const double* cs, double cw, double (*red)[2][NA], double (*ms)[NA])
{
    const int slot = threadIdx.x & (kRowSlots - 1), lane = threadIdx.x & 31, warp = threadIdx.x >> 5;
    RowWalk w(slot * VEC, kRowSlots * VEC, uint32_t(Nv));
    auto warp_sums = [&](double (&m)[NA], int r) {
#pragma unroll
        for (int i = 0; i < NA; ++i) {
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) m[i] += __shfl_xor_sync(0xffffffffu, m[i], o);
        }
        if (lane == 0) {
#pragma unroll
            for (int i = 0; i < NA; ++i) red[slot >> 5][r][i] = m[i];
        }
    };
    if (blockDim.x > kRowSlots) {
        const int r = threadIdx.x >= kRowSlots;
        const T* row = r ? r1 : r0;
        if (row) {
            double m[NA];
#pragma unroll
            for (int i = 0; i < NA; ++i) m[i] = 0.0;
#pragma unroll 4
            for (int v = slot * VEC; v < n; v += kRowSlots * VEC) {
                Chunk<T, VEC> a;
                a.load(row + v);
                chunk_moments<T, VEC, NA>(a, cs[w.ix], cs[w.iy], cs + w.iz, m);
                w.next();
            }
            warp_sums(m, r);
        }
    } else {
        double m0[NA], m1[NA];
#pragma unroll
        for (int i = 0; i < NA; ++i) m0[i] = m1[i] = 0.0;
#pragma unroll 2
        for (int v = slot * VEC; v < n; v += kRowSlots * VEC) {
            Chunk<T, VEC> a, b;
            if (r0) a.load(r0 + v);
            if (r1) b.load(r1 + v);
            if (r0) chunk_moments<T, VEC, NA>(a, cs[w.ix], cs[w.iy], cs + w.iz, m0);
            if (r1) chunk_moments<T, VEC, NA>(b, cs[w.ix], cs[w.iy], cs + w.iz, m1);
            w.next();
        }
        if (r0) warp_sums(m0, 0);
        if (r1) warp_sums(m1, 1);
    }
    __syncthreads();
    if (warp == 0 && lane < NA) {
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            double s = 0.0;
            for (int k = 0; k < kRowWarps; ++k) s += red[k][r][lane];
            ms[r][lane] = s * cw;
        }
    }
    __syncwarp();
}

// moment rows alone (the same sums, in the same order, as inside the stage kernels)
template <typename T, int VEC, int NA>
__global__ void __launch_bounds__(kRowSlots) row_moments_kernel(const T* __restrict__ f, int Nv, const double* c0, double cw,
                                                          double* __restrict__ U)
{
    __shared__ double red[kRowWarps][2][NA];
    __shared__ double ms[2][NA];
    __shared__ double cs[kMaxNv];
    const int64_t dof = blockIdx.x;
    const int n = Nv * Nv * Nv;
    for (int i = threadIdx.x; i < Nv; i += blockDim.x) cs[i] = c0[i];
    __syncthreads();
    two_row_moments<T, VEC, NA>(f + dof * int64_t(n), nullptr, n, Nv, cs, cw, red, ms);
    if (threadIdx.x < NA) U[dof * NA + threadIdx.x] = ms[0][threadIdx.x];
}

// temperature-dependent collision frequency of a moment row
__device__ __forceinline__ double collision_rate(const double* u, double prefac, double omega)
{
    double rho, ux, uy, uz, Tt;
    const double u5[5] = {u[0], u[1], u[2], u[3], u[4]};
    row_state(u5, rho, ux, uy, uz, Tt);
    return prefac * rho * pow(Tt, 1.0 - omega);
}

// Parameters of one relaxation target: u and 1/T of the separable exponentials,
// the leading factor, and the ES tensor's or the Shakov polynomial's numbers
struct Target {
    double u[3], it, am, p[10];
};

template <int NA>
__device__ __forceinline__ void target_params(const double* u, double Pr, Target& t)
{
    if constexpr (NA == 11) {
        double g[10];
        es_params(u, Pr, g);
#pragma unroll
        for (int i = 0; i < 10; ++i) t.p[i] = g[i];
    } else {
        double rho, T;
        const double u5[5] = {u[0], u[1], u[2], u[3], u[4]};
        row_state(u5, rho, t.u[0], t.u[1], t.u[2], T);
        const double pt = kPi * T;
        t.am = rho / (pt * sqrt(pt));
        t.it = 1.0 / T;
        if constexpr (NA == 14) {
            double s[7];
            shakov_params(u, Pr, s);
#pragma unroll
            for (int i = 0; i < 7; ++i) t.p[i] = s[i];
        }
    }
}

// exponential tables of the targets (NA != 11), all threads
__device__ __forceinline__ void target_tables(const Target* t, int nt, int Nv, const double* cs,
                                              double (*ex)[3][kMaxNv])
{
    for (int i = threadIdx.x; i < nt * 3 * Nv; i += blockDim.x) {
        const int j = i / (3 * Nv), r = i - j * 3 * Nv, d = r / Nv, k = r - d * Nv;
        const double c = cs[k] - t[j].u[d];
        ex[j][d][k] = exp(-c * c * t[j].it);
    }
}

template <int NA>
__device__ __forceinline__ double target_at(const Target& t, const double (*ex)[kMaxNv], const double* cs, uint32_t ix,
                                            uint32_t iy, uint32_t iz)
{
    if constexpr (NA == 11) {
        return es_eval(t.p, cs[ix], cs[iy], cs[iz]);
    } else {
        const double m = t.am * ex[0][ix] * ex[1][iy] * ex[2][iz];
        if constexpr (NA == 14) return m * shakov_factor(t.p, cs[ix], cs[iy], cs[iz]);
        else return m;
    }
}

// NA = 5: BGK (separable Maxwellians); NA = 11: ES-BGK (second moments
// relaxed implicitly at nu/Pr, Gaussians evaluated per velocity); NA = 14:
// Shakov (second moments at nu, heat flux at nu Pr, separable Maxwellians
// times the heat-flux polynomial).
// AR > 0: the stage at compile time, so that a thread has all 2 AR rows of a
// chunk (of two chunks for AR <= 2) in flight at once; AR = 0 reads the stage
// from the arguments.  The moment algebra (pow, divisions) runs in one warp, a
// lane per implicit stage, instead of in every thread.  Bound: the
// latency of HBM loads (0.65 of the copy rate at 28 warps an SM; conversions 29 %,
// FP64 20 %).
template <typename T, int VEC, int NA, int AR>
__global__ void __launch_bounds__(512, NA == 5 && AR <= 2 ? 2 : 1) ars_kernel(const bdgfs_ars_args g)
{
    __shared__ double red[kRowWarps][2][NA];
    __shared__ double ms[2][NA];                       // moments of f_0 and of L_{ar-1}
    __shared__ double cs[kMaxNv];
    __shared__ double ex[NA == 11 ? 1 : 4][3][kMaxNv];
    __shared__ Target tg[4];
    __shared__ double nu[4];
    const int64_t dof = blockIdx.x;
    const int Nv = g.Nv, ar = AR > 0 ? AR : g.stage, flags = g.flags;
    const int n = Nv * Nv * Nv;
    const int64_t off = dof * int64_t(n);
    for (int i = threadIdx.x; i < Nv; i += blockDim.x) cs[i] = g.c0[i];
    __syncthreads();
    // ---- moments of f_0 and of the newest explicit part L_{ar-1}
    const T* r0 = flags & BDGFS_ARS_MOM0 ? static_cast<const T*>(g.f[0]) + off : nullptr;
    const T* r1 = flags & BDGFS_ARS_MOML ? static_cast<const T*>(g.L[ar - 1]) + off : nullptr;
    if (r0 || r1) two_row_moments<T, VEC, NA>(r0, r1, n, Nv, cs, g.cw, red, ms);
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        if (lane < NA) {
            if (r0) g.U[0][dof * NA + lane] = ms[0][lane];
            if (r1) g.LU[ar - 1][dof * NA + lane] = ms[1][lane];
        }
        __syncwarp();
        // lane j - 1 holds moment row U_j, j = 1..ar (further lanes repeat U_ar).
        // Stage moments: U_ar = U_0 + dt sum_j ae_j LU_j (the relaxation
        // conserves the first five); higher moments relax implicitly
        const int j = min(lane + 1, ar);
        if (flags & (BDGFS_ARS_MOMU | BDGFS_ARS_DIST)) {
            double u[NA];
#pragma unroll
            for (int i = 0; i < NA; ++i) {
                if (j < ar || !(flags & BDGFS_ARS_MOMU)) {
                    // U_j of the implicit parts: needed for the target, and for
                    // the higher moments' history
                    u[i] = (flags & BDGFS_ARS_DIST) || NA > 5 || j == ar ? g.U[j][dof * NA + i] : 0.0;
                } else {
                    double s = r0 ? ms[0][i] : g.U[0][dof * NA + i];
                    for (int k = 0; k < ar; ++k)
                        s += g.dt * g.ae[k] * (k == ar - 1 && r1 ? ms[1][i] : g.LU[k][dof * NA + i]);
                    u[i] = s;
                }
            }
            double rate = 0.0;
            if (NA > 5 || (flags & BDGFS_ARS_DIST)) rate = collision_rate(u, g.prefac, g.omega);
            if constexpr (NA >= 11) {
                if (flags & BDGFS_ARS_MOMU) {
                    // second moments: rate nu/Pr (ES-BGK) or nu (Shakov) towards the Maxwellian's
                    const double w = g.ai[j - 1] * g.dt * rate, w2 = NA == 11 ? w / g.Pr : w;
                    double t[6];
                    maxwell_second(u, t);
#pragma unroll
                    for (int k = 0; k < 6; ++k) {
                        const double part = w2 * (t[k] - u[5 + k]);
                        double num = u[5 + k];
                        for (int q = 1; q < ar; ++q) num += __shfl_sync(0xffffffffu, part, q - 1);
                        if (j == ar) u[5 + k] = (num + w2 * t[k]) / (1.0 + w2);
                    }
                    if constexpr (NA == 14) {
                        // heat flux: dQ/dt = nu (Q(M) + (1 - Pr)(q - Q) - Pr Q), -Pr Q implicit
                        double h[3];
                        shakov_heat(u, g.Pr, h);
#pragma unroll
                        for (int k = 0; k < 3; ++k) {
                            const double part = w * (h[k] - g.Pr * u[11 + k]);
                            double num = u[11 + k];
                            for (int q = 1; q < ar; ++q) num += __shfl_sync(0xffffffffu, part, q - 1);
                            if (j == ar) u[11 + k] = (num + w * h[k]) / (1.0 + g.Pr * w);
                        }
                    }
                }
            }
            if (lane == ar - 1 && (flags & BDGFS_ARS_MOMU)) {
#pragma unroll
                for (int i = 0; i < NA; ++i) g.U[ar][dof * NA + i] = u[i];
            }
            if (lane < ar && (flags & BDGFS_ARS_DIST)) {
                nu[lane] = rate;
                target_params<NA>(u, g.Pr, tg[lane]);
            }
        }
    }
    if (!(flags & BDGFS_ARS_DIST)) return;
    __syncthreads();
    if constexpr (NA != 11) {
        target_tables(tg, ar, Nv, cs, ex);
        __syncthreads();
    }

    const double dt = g.dt;
    const double aii = g.ai[ar - 1] * dt * nu[ar - 1];
    const double inv = 1.0 / (1.0 + aii);
    const T* f0 = static_cast<const T*>(g.f[0]) + off;
    T* fout = static_cast<T*>(g.fout) + off;
    auto finish = [&](int v, const RowWalk& w, double (&acc)[VEC]) {
        Chunk<T, VEC> o;
#pragma unroll
        for (int q = 0; q < VEC; ++q)
            o.v[q] = T((acc[q] + aii * target_at<NA>(tg[ar - 1], ex[NA == 11 ? 0 : ar - 1], cs, w.ix, w.iy, w.iz + q)) * inv);
        o.store(fout + v);
    };
    auto add_l = [&](int j, const Chunk<T, VEC>& c, double (&acc)[VEC]) {
        const double w = g.ae[j] * dt;
#pragma unroll
        for (int q = 0; q < VEC; ++q) acc[q] += w * double(c.v[q]);
    };
    auto add_f = [&](int j, const Chunk<T, VEC>& c, const RowWalk& x, double (&acc)[VEC]) {
        const double w = g.ai[j - 1] * dt * nu[j - 1];
#pragma unroll
        for (int q = 0; q < VEC; ++q)
            acc[q] += w * (target_at<NA>(tg[j - 1], ex[NA == 11 ? 0 : j - 1], cs, x.ix, x.iy, x.iz + q) - double(c.v[q]));
    };
    RowWalk w(threadIdx.x * VEC, blockDim.x * VEC, uint32_t(Nv));
    if constexpr (AR > 0) {
        const T* L[AR];
        const T* F[AR];
#pragma unroll
        for (int j = 0; j < AR; ++j) {
            L[j] = static_cast<const T*>(g.L[j]) + off;
            F[j] = j ? static_cast<const T*>(g.f[j]) + off : f0;
        }
        auto step = [&](int v, const Chunk<T, VEC> (&cf)[AR], const Chunk<T, VEC> (&cl)[AR]) {
            double acc[VEC];
#pragma unroll
            for (int q = 0; q < VEC; ++q) acc[q] = double(cf[0].v[q]);
#pragma unroll
            for (int j = 0; j < AR; ++j) add_l(j, cl[j], acc);
#pragma unroll
            for (int j = 1; j < AR; ++j) add_f(j, cf[j], w, acc);
            finish(v, w, acc);
            w.next();
        };
        constexpr int U = AR <= 2 ? 2 : 1;             // chunks in flight
        const int st = int(blockDim.x) * VEC;
        for (int v = threadIdx.x * VEC; v < n; v += U * st) {
            Chunk<T, VEC> cf[U][AR], cl[U][AR];
#pragma unroll
            for (int k = 0; k < U; ++k) {
                if (v + k * st < n) {
#pragma unroll
                    for (int j = 0; j < AR; ++j) {
                        cf[k][j].load(F[j] + v + k * st);
                        cl[k][j].load(L[j] + v + k * st);
                    }
                }
            }
#pragma unroll
            for (int k = 0; k < U; ++k)
                if (v + k * st < n) step(v + k * st, cf[k], cl[k]);
        }
    } else {
        for (int v = threadIdx.x * VEC; v < n; v += blockDim.x * VEC) {
            double acc[VEC];
            Chunk<T, VEC> c;
            c.load(f0 + v);
#pragma unroll
            for (int q = 0; q < VEC; ++q) acc[q] = double(c.v[q]);
            for (int j = 0; j < ar; ++j) {
                c.load(static_cast<const T*>(g.L[j]) + off + v);
                add_l(j, c, acc);
            }
            for (int j = 1; j < ar; ++j) {
                c.load(static_cast<const T*>(g.f[j]) + off + v);
                add_f(j, c, w, acc);
            }
            finish(v, w, acc);
            w.next();
        }
    }
}

// One IMEX-BDF step (updateMom{q}_BDF + constructMaxwellian +
// updateDistribution{q}_BDF): with N = -sum_i (a_i X_i + g_i dt LX_i),
//   U  = N / a_q for the conserved five; higher moments relax implicitly
//        (ES-BGK second moments at b nu/Pr, Shakov second moments at b nu and
//        the heat flux with denominator a_q + Pr b dt nu)
//   f  = (N_f + b dt nu M[U]) / (a_q + b dt nu).
// One CTA per distribution; the newest moment rows (of f_{q-1} and of
// L_{q-1}) are reduced in the same launch when BDGFS_BDF_MOMN is set.  BQ > 0:
// the order q at compile time (all 2 q rows of a chunk in flight); BQ = 0 reads
// it from the arguments.  Moment algebra in one thread.  315 rows of 24^3 FP32,
// Shakov, BDF-2, one B200: 86 -> 53 us (512 threads a row), 45 with a row per half
// of them.  Bound: 116 registers leave one CTA an SM, so its barriers and loads show.
template <typename T, int VEC, int NA, int BQ>
__global__ void __launch_bounds__(512, NA == 5 ? 2 : 1) bdf_kernel(const bdgfs_bdf_args g)
{
    __shared__ double red[kRowWarps][2][NA];
    __shared__ double ms[2][NA];                       // moments of f_{q-1} and of L_{q-1}
    __shared__ double cs[kMaxNv];
    __shared__ double ex[1][3][kMaxNv];
    __shared__ Target tg;
    __shared__ double nu;
    const int64_t dof = blockIdx.x;
    const int Nv = g.Nv, q = BQ > 0 ? BQ : g.q, flags = g.flags;
    const int n = Nv * Nv * Nv;
    const int64_t off = dof * int64_t(n);
    for (int i = threadIdx.x; i < Nv; i += blockDim.x) cs[i] = g.c0[i];
    __syncthreads();
    const bool momn = flags & BDGFS_BDF_MOMN;
    if (momn)
        two_row_moments<T, VEC, NA>(static_cast<const T*>(g.f[q - 1]) + off, static_cast<const T*>(g.L[q - 1]) + off, n,
                                    Nv, cs, g.cw, red, ms);
    const double aq = g.a[q];
    if (threadIdx.x < 32) {
        const int lane = threadIdx.x;
        if (momn && lane < NA) {
            g.U[q - 1][dof * NA + lane] = ms[0][lane];
            g.LU[q - 1][dof * NA + lane] = ms[1][lane];
        }
        __syncwarp();
        if (flags & (BDGFS_BDF_MOMU | BDGFS_BDF_DIST)) {
            // lane k forms N_k (or reads U_k), then lane 0 has the row
            double u[NA];
            const int k = min(lane, NA - 1);
            double s = 0.0;
            if (flags & BDGFS_BDF_MOMU) {
                for (int i = 0; i < q; ++i) {
                    const bool fresh = i == q - 1 && momn;
                    const double ui = fresh ? ms[0][k] : g.U[i][dof * NA + k];
                    const double li = fresh ? ms[1][k] : g.LU[i][dof * NA + k];
                    s -= g.a[i] * ui + g.g[i] * g.dt * li;
                }
            } else {
                s = g.Unew[dof * NA + k];
            }
#pragma unroll
            for (int i = 0; i < NA; ++i) u[i] = __shfl_sync(0xffffffffu, s, i);
            if (lane == 0) {
                if (flags & BDGFS_BDF_MOMU) {
#pragma unroll
                    for (int i = 0; i < 5; ++i) u[i] = u[i] / aq;
                }
                double rate = 0.0;
                if (NA > 5 || (flags & BDGFS_BDF_DIST)) rate = collision_rate(u, g.prefac, g.omega);
                if (flags & BDGFS_BDF_MOMU) {
                    if constexpr (NA >= 11) {
                        const double w = g.b * g.dt * rate * (NA == 11 ? 1.0 / g.Pr : 1.0);
                        double t[6];
                        maxwell_second(u, t);
#pragma unroll
                        for (int i = 0; i < 6; ++i) u[5 + i] = (u[5 + i] + w * t[i]) / (aq + w);
                    }
                    if constexpr (NA == 14) {
                        const double w = g.b * g.dt * rate;
                        double h[3];
                        shakov_heat(u, g.Pr, h);
#pragma unroll
                        for (int i = 0; i < 3; ++i) u[11 + i] = (u[11 + i] + w * h[i]) / (aq + g.Pr * w);
                    }
#pragma unroll
                    for (int i = 0; i < NA; ++i) g.Unew[dof * NA + i] = u[i];
                }
                if (flags & BDGFS_BDF_DIST) {
                    nu = rate;
                    target_params<NA>(u, g.Pr, tg);
                }
            }
        }
    }
    if (!(flags & BDGFS_BDF_DIST)) return;
    __syncthreads();
    if constexpr (NA != 11) {
        target_tables(&tg, 1, Nv, cs, ex);
        __syncthreads();
    }
    const double bdn = g.b * g.dt * nu;
    const double inv = 1.0 / (aq + bdn);
    T* fout = static_cast<T*>(g.fout) + off;
    RowWalk w(threadIdx.x * VEC, blockDim.x * VEC, uint32_t(Nv));
    constexpr int QB = BQ > 0 ? BQ : 1;
    for (int v = threadIdx.x * VEC; v < n; v += blockDim.x * VEC) {
        double acc[VEC];
#pragma unroll
        for (int j = 0; j < VEC; ++j) acc[j] = 0.0;
        auto add = [&](int i, const Chunk<T, VEC>& cf, const Chunk<T, VEC>& cl) {
            const double wa = g.a[i], wg = g.g[i] * g.dt;
#pragma unroll
            for (int j = 0; j < VEC; ++j) acc[j] -= wa * double(cf.v[j]) + wg * double(cl.v[j]);
        };
        if constexpr (BQ > 0) {
            Chunk<T, VEC> cf[QB], cl[QB];
#pragma unroll
            for (int i = 0; i < QB; ++i) {
                cf[i].load(static_cast<const T*>(g.f[i]) + off + v);
                cl[i].load(static_cast<const T*>(g.L[i]) + off + v);
            }
#pragma unroll
            for (int i = 0; i < QB; ++i) add(i, cf[i], cl[i]);
        } else {
            for (int i = 0; i < q; ++i) {
                Chunk<T, VEC> cf, cl;
                cf.load(static_cast<const T*>(g.f[i]) + off + v);
                cl.load(static_cast<const T*>(g.L[i]) + off + v);
                add(i, cf, cl);
            }
        }
        Chunk<T, VEC> o;
#pragma unroll
        for (int j = 0; j < VEC; ++j)
            o.v[j] = T((acc[j] + bdn * target_at<NA>(tg, ex[0], cs, w.ix, w.iy, w.iz + j)) * inv);
        o.store(fout + v);
        w.next();
    }
}

}  // namespace bdgfs

using namespace bdgfs;

namespace {

bool a16(const void* p) { return (reinterpret_cast<uintptr_t>(p) & 15u) == 0; }

template <typename K4, typename K1, typename... Args>
int32_t launch_rows(bool v4, K4 k4, K1 k1, int64_t ndof, cudaStream_t st, Args... args)
{
    if (v4)
        k4<<<unsigned(ndof), 256, 0, st>>>(args...);
    else
        k1<<<unsigned(ndof), 256, 0, st>>>(args...);
    return cuda_status(cudaGetLastError());
}

// Relaxation kernels: 512 threads per row when the rows are too few to fill
// the SMs with 256 (fewer than four CTAs each), else 256
unsigned relax_threads(int64_t ndof) { return ndof < 148 * 4 ? 512 : 256; }

template <typename K, typename A>
int32_t launch_relax(K k, const A& a, cudaStream_t st)
{
    k<<<unsigned(a.ndof), relax_threads(a.ndof), 0, st>>>(a);
    return cuda_status(cudaGetLastError());
}

template <int NA>
int32_t launch_moments(const void* f, int64_t ndof, int Nv, int fp64, const double* c0, double cw, double* U,
                       cudaStream_t st)
{
    const bool v4 = Nv % 4 == 0 && a16(f);
#define GO(T, V) row_moments_kernel<T, V, NA><<<unsigned(ndof), kRowSlots, 0, st>>>(static_cast<const T*>(f), Nv, c0, cw, U)
    if (fp64) {
        if (v4) GO(double, 4);
        else GO(double, 1);
    } else {
        if (v4) GO(float, 4);
        else GO(float, 1);
    }
#undef GO
    return cuda_status(cudaGetLastError());
}

template <typename T, int NA>
int32_t launch_ars(bool v4, const bdgfs_ars_args& a, cudaStream_t st)
{
    if (v4) {
        if (a.stage == 1) return launch_relax(ars_kernel<T, 4, NA, 1>, a, st);
        if (a.stage == 2) return launch_relax(ars_kernel<T, 4, NA, 2>, a, st);
        if (a.stage == 3) return launch_relax(ars_kernel<T, 4, NA, 3>, a, st);
        return launch_relax(ars_kernel<T, 4, NA, 4>, a, st);
    }
    return launch_relax(ars_kernel<T, 1, NA, 0>, a, st);
}

template <typename T, int NA>
int32_t launch_bdf(bool v4, const bdgfs_bdf_args& a, cudaStream_t st)
{
    if (v4 && a.q == 2) return launch_relax(bdf_kernel<T, 4, NA, 2>, a, st);
    if (v4 && a.q == 3) return launch_relax(bdf_kernel<T, 4, NA, 3>, a, st);
    if (v4) return launch_relax(bdf_kernel<T, 4, NA, 0>, a, st);
    return launch_relax(bdf_kernel<T, 1, NA, 0>, a, st);
}

}  // namespace

extern "C" int32_t bdgfs_bgk_moments(const void* f, int64_t ndof, int32_t Nv, int32_t fp64, const double* c0,
                                     double cw, double* U, void* stream)
{
    if (!f || !c0 || !U || ndof < 0 || ndof > 2147483647LL || Nv < 1 || Nv > kMaxNv) return BDGFS_EINVAL;
    if (ndof == 0) return BDGFS_OK;
    return launch_moments<5>(f, ndof, Nv, fp64, c0, cw, U, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t bdgfs_bgk_maxwellian(const double* U, int64_t ndof, int32_t Nv, int32_t fp64,
                                        const double* c0, void* M, void* stream)
{
    if (!U || !c0 || !M || ndof < 0 || ndof > 2147483647LL || Nv < 1 || Nv > kMaxNv) return BDGFS_EINVAL;
    if (ndof == 0) return BDGFS_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool v4 = Nv % 4 == 0 && a16(M);
    if (fp64)
        return launch_rows(v4, bgk_maxwellian_kernel<double, 4>, bgk_maxwellian_kernel<double, 1>, ndof, st, U,
                           int(Nv), c0, static_cast<double*>(M));
    return launch_rows(v4, bgk_maxwellian_kernel<float, 4>, bgk_maxwellian_kernel<float, 1>, ndof, st, U,
                       int(Nv), c0, static_cast<float*>(M));
}

extern "C" int32_t bdgfs_ars_stage(const bdgfs_ars_args* a, void* stream)
{
    if (!a || !a->c0 || a->ndof < 0 || a->ndof > 2147483647LL || a->Nv < 1 || a->Nv > kMaxNv ||
        a->stage < 1 || a->stage > 4 || (a->flags & ~15) ||
        (a->model != BDGFS_ARS_BGK && a->model != BDGFS_ARS_ESBGK && a->model != BDGFS_ARS_SHAKOV) ||
        (a->model != BDGFS_ARS_BGK && !(a->Pr > 0.0)))
        return BDGFS_EINVAL;
    const int ar = a->stage, fl = a->flags;
    bool ok = true, v4 = a->Nv % 4 == 0;
    if (fl & BDGFS_ARS_MOM0) ok = ok && a->f[0] && a->U[0];
    if (fl & BDGFS_ARS_MOML) ok = ok && a->L[ar - 1] && a->LU[ar - 1];
    if (fl & BDGFS_ARS_MOMU) {
        ok = ok && a->U[0] && a->U[ar];
        for (int j = 0; j < ar; ++j) ok = ok && a->LU[j];
    }
    if (fl & BDGFS_ARS_DIST) {
        ok = ok && a->fout && a->f[0];
        for (int j = 0; j < ar; ++j) ok = ok && a->L[j] && (j == 0 || a->f[j]);
        for (int j = 1; j <= ar; ++j) ok = ok && a->U[j];
        v4 = v4 && a16(a->fout);
    }
    if (!ok) return BDGFS_EINVAL;
    for (int j = 0; j < ar; ++j) {
        if (a->f[j]) v4 = v4 && a16(a->f[j]);
        if (a->L[j]) v4 = v4 && a16(a->L[j]);
    }
    if (a->ndof == 0) return BDGFS_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define ARS_GO(NA) return a->fp64 ? launch_ars<double, NA>(v4, *a, st) : launch_ars<float, NA>(v4, *a, st);
    if (a->model == BDGFS_ARS_SHAKOV) { ARS_GO(14) }
    if (a->model == BDGFS_ARS_ESBGK) { ARS_GO(11) }
    ARS_GO(5)
#undef ARS_GO
}

extern "C" int32_t bdgfs_esbgk_moments(const void* f, int64_t ndof, int32_t Nv, int32_t fp64,
                                       const double* c0, double cw, double* U, void* stream)
{
    if (!f || !c0 || !U || ndof < 0 || ndof > 2147483647LL || Nv < 1 || Nv > kMaxNv) return BDGFS_EINVAL;
    if (ndof == 0) return BDGFS_OK;
    return launch_moments<11>(f, ndof, Nv, fp64, c0, cw, U, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t bdgfs_esbgk_gaussian(const double* U, int64_t ndof, int32_t Nv, int32_t fp64,
                                        const double* c0, double Pr, void* M, void* stream)
{
    if (!U || !c0 || !M || ndof < 0 || ndof > 2147483647LL || Nv < 1 || Nv > kMaxNv || !(Pr > 0.0))
        return BDGFS_EINVAL;
    if (ndof == 0) return BDGFS_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool v4 = Nv % 4 == 0 && a16(M);
    if (fp64)
        return launch_rows(v4, esbgk_gaussian_kernel<double, 4>, esbgk_gaussian_kernel<double, 1>, ndof, st, U,
                           int(Nv), c0, Pr, static_cast<double*>(M));
    return launch_rows(v4, esbgk_gaussian_kernel<float, 4>, esbgk_gaussian_kernel<float, 1>, ndof, st, U,
                       int(Nv), c0, Pr, static_cast<float*>(M));
}

extern "C" int32_t bdgfs_shakov_moments(const void* f, int64_t ndof, int32_t Nv, int32_t fp64,
                                        const double* c0, double cw, double* U, void* stream)
{
    if (!f || !c0 || !U || ndof < 0 || ndof > 2147483647LL || Nv < 1 || Nv > kMaxNv) return BDGFS_EINVAL;
    if (ndof == 0) return BDGFS_OK;
    return launch_moments<14>(f, ndof, Nv, fp64, c0, cw, U, static_cast<cudaStream_t>(stream));
}

extern "C" int32_t bdgfs_shakov_target(const double* U, int64_t ndof, int32_t Nv, int32_t fp64,
                                       const double* c0, double Pr, void* S, void* stream)
{
    if (!U || !c0 || !S || ndof < 0 || ndof > 2147483647LL || Nv < 1 || Nv > kMaxNv || !(Pr > 0.0))
        return BDGFS_EINVAL;
    if (ndof == 0) return BDGFS_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
    const bool v4 = Nv % 4 == 0 && a16(S);
    if (fp64)
        return launch_rows(v4, shakov_target_kernel<double, 4>, shakov_target_kernel<double, 1>, ndof, st, U,
                           int(Nv), c0, Pr, static_cast<double*>(S));
    return launch_rows(v4, shakov_target_kernel<float, 4>, shakov_target_kernel<float, 1>, ndof, st, U,
                       int(Nv), c0, Pr, static_cast<float*>(S));
}

extern "C" int32_t bdgfs_bdf_step(const bdgfs_bdf_args* a, void* stream)
{
    if (!a || a->ndof < 0 || a->ndof > 2147483647LL || a->Nv < 1 || a->Nv > kMaxNv || !a->c0 ||
        a->q < 1 || a->q > 3 || (a->flags & ~7) || !a->Unew ||
        (a->model != BDGFS_ARS_BGK && a->model != BDGFS_ARS_ESBGK && a->model != BDGFS_ARS_SHAKOV) ||
        (a->model != BDGFS_ARS_BGK && !(a->Pr > 0.0)) || a->a[a->q] == 0.0)
        return BDGFS_EINVAL;
    const int q = a->q;
    if (a->flags & BDGFS_BDF_MOMN) {
        if (!a->f[q - 1] || !a->L[q - 1] || !a->U[q - 1] || !a->LU[q - 1]) return BDGFS_EINVAL;
    }
    if (a->flags & BDGFS_BDF_MOMU) {
        for (int i = 0; i < q; ++i)
            if (!a->U[i] || !a->LU[i]) return BDGFS_EINVAL;
    }
    bool v4 = a->Nv % 4 == 0;
    if (a->flags & BDGFS_BDF_DIST) {
        if (!a->fout) return BDGFS_EINVAL;
        v4 = v4 && a16(a->fout);
        for (int i = 0; i < q; ++i) {
            if (!a->f[i] || !a->L[i]) return BDGFS_EINVAL;
            v4 = v4 && a16(a->f[i]) && a16(a->L[i]);
        }
    } else if (a->flags & BDGFS_BDF_MOMN) {
        v4 = v4 && a16(a->f[q - 1]) && a16(a->L[q - 1]);
    }
    if (a->ndof == 0) return BDGFS_OK;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define BDF_GO(NA) return a->fp64 ? launch_bdf<double, NA>(v4, *a, st) : launch_bdf<float, NA>(v4, *a, st);
    if (a->model == BDGFS_ARS_SHAKOV) { BDF_GO(14) }
    if (a->model == BDGFS_ARS_ESBGK) { BDF_GO(11) }
    BDF_GO(5)
#undef BDF_GO
}
