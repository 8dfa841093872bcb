// FR residual of affine tensor-product elements, by lines and inflow faces.
//
// Same operator as bdgfs_fr_rhs_tensor (fr.cu): R = M1 F~ + M3 (F^n - M2 F~).
// On an affine element the metric is one matrix S per element, so with
// al_d = sum_k S[d][k] c_k
//   M1 F~          = sum_d al_d D_d u               (D: the 1-D derivative along d-lines)
//   |n| n.c        = -+ al_d on the lower / upper face of direction d
//   F^n - M2 F~    = |n| n.c (u_R - u_L) where n.c < 0, else 0  (upwind flux)
//                  = -|al_d| (u_R - u_L) on the inflow face, 0 on the other
// and M3 factors into the tangential quadrature KW (per face axis) and the
// normal values kn of the lifting.  A velocity sees one of the two faces of each
// direction, so a thread loads P^(ND-1) neighbour values per direction instead of
// two faces' own and neighbour values, and lifts with 1-D factors: for hex P2
// 27 u, 27 neighbour and the combination rows instead of 216 rows, and about 620
// FMAs a velocity and element instead of 2270.  Measured on one B200, 24^3 FP32
// (bdgfs_fr_rhs_tensor -> this): RK stage of 210 hexes P2 593 -> 344 us (3.7 TB/s
// of u, x1, x2 and out), L(u) of 128 quads P3 125 -> 61 us (3.7 TB/s).  Bound: the
// latency of the dependent loads (u, three faces, x1, x2) at 16 warps an SM (0.59 of
// the copy rate), and instruction fetch of the unrolled body.
//
// A thread holds all solution points of an element at VB consecutive velocities
// in registers: u, R and one direction's neighbours, loaded one direction ahead (FP32
// hex P2 without spills; 284 bytes of them on hex P1 at four velocities, 548 on hex P2
// in FP64).
// Lanes choose their inflow face by a pointer select (two table entries a warp);
// velocities of a chunk that disagree about the face take both.
#include <algorithm>
#include <type_traits>

#include "fr_common.cuh"

namespace bdgfs {

template <typename T, int ND, int P>
struct AffArgs {
    bdgfs_fr_eles el;
    bdgfs_fr_walls wl;
    const T* u;
    const T* uf;                 // face values, or null: neighbours read from u through fsel
    const int32_t* fsel;
    const int32_t* fid;          // [2 ND][P^(ND-1)]
    const T* smat;               // [E][ND][ND]
    T* out;
    const T *x1, *x2;
    T a, b, c1, c2;
    T D[P][P], KW[P][P], kn[2][P];
    int64_t chunk;
};

// points of a d-line: stride st; base of line t (tangential index, first
// remaining axis fastest)
template <int ND, int P>
__host__ __device__ constexpr int line_base(int d, int t)
{
    if (ND == 2) return d == 0 ? t * P : t;
    const int t0 = t % P, t1 = t / P;
    return d == 0 ? t0 * P + t1 * P * P : (d == 1 ? t0 + t1 * P * P : t0 + t1 * P);
}

template <int ND, int P>
struct AffShape {
    static constexpr int NF1 = ND == 3 ? P * P : P, NU = NF1 * P, NF = 2 * ND * NF1;
};

// R (+)= al D u along direction d
template <int d, typename T, int ND, int P, int VB>
__device__ __forceinline__ void aff_volume(const AffArgs<T, ND, P>& g, const Vec<T, VB> (&u)[AffShape<ND, P>::NU],
                                           const T (&al)[VB], T (&R)[AffShape<ND, P>::NU][VB])
{
    constexpr int NF1 = AffShape<ND, P>::NF1;
    constexpr int st = d == 0 ? 1 : (d == 1 ? P : P * P);
#pragma unroll
    for (int t = 0; t < NF1; ++t) {
        const int b = line_base<ND, P>(d, t);
#pragma unroll
        for (int i = 0; i < P; ++i)
#pragma unroll
            for (int q = 0; q < VB; ++q) {
                T y = g.D[i][0] * u[b].v[q];
#pragma unroll
                for (int j = 1; j < P; ++j) y += g.D[i][j] * u[b + j * st].v[q];
                if (d == 0) R[b + i * st][q] = al[q] * y;
                else R[b + i * st][q] += al[q] * y;
            }
    }
}

// lifting of -|al| (u_R - u_L) on face (d, s), for the velocities that flow in
// there; wk, wsc, wu: the face table
template <int d, typename T, int ND, int P, int VB>
__device__ __forceinline__ void aff_lift(const AffArgs<T, ND, P>& g, const T (&S)[ND][ND], const T (&c)[VB][3], int s,
                                         const signed char* wk, const T* wsc, const T (*wu)[3],
                                         Vec<T, VB> (&ur)[AffShape<ND, P>::NF1],
                                         const Vec<T, VB> (&u)[AffShape<ND, P>::NU], const T (&al)[VB],
                                         T (&R)[AffShape<ND, P>::NU][VB])
{
    constexpr int NF1 = AffShape<ND, P>::NF1;
    constexpr int st = d == 0 ? 1 : (d == 1 ? P : P * P);
    const int i0 = (2 * d + s) * NF1;
    T w[VB];
#pragma unroll
    for (int q = 0; q < VB; ++q) w[q] = s ? min(al[q], T(0)) : -max(al[q], T(0));
    T J[NF1][VB];
#pragma unroll
    for (int t = 0; t < NF1; ++t) {
        const int b = line_base<ND, P>(d, t);
        const int kd = wk[i0 + t];
        if (kd >= 0) {
            if (kd == BDGFS_BC_SPECULAR_Z) {                 // the mirrored chunk comes reversed
#pragma unroll
                for (int q = 0; q < VB / 2; ++q) {
                    const T x = ur[t].v[q];
                    ur[t].v[q] = ur[t].v[VB - 1 - q];
                    ur[t].v[VB - 1 - q] = x;
                }
            }
#pragma unroll
            for (int q = 0; q < VB; ++q) {
                const T ul = s ? u[b + (P - 1) * st].v[q] : u[b].v[q];
                if (kd < BDGFS_BC_OUTLET) {                  // diffuse wall or inlet
                    T fac = T(0);
#pragma unroll
                    for (int k = 0; k < ND; ++k) fac += (c[q][k] - wu[i0 + t][k]) * S[d][k];
                    const bool in = s ? fac < T(0) : fac > T(0);
                    ur[t].v[q] = in ? ur[t].v[q] * wsc[i0 + t] : ul;
                } else if (kd == BDGFS_BC_OUTLET) {
                    ur[t].v[q] = ul;
                }
            }
        }
#pragma unroll
        for (int q = 0; q < VB; ++q) {
            const T ul = s ? u[b + (P - 1) * st].v[q] : u[b].v[q];
            J[t][q] = w[q] * (ur[t].v[q] - ul);
        }
    }
    // tangential quadrature, axis by axis
#pragma unroll
    for (int ax = 0; ax < ND - 1; ++ax) {
        const int ts = ax == 0 ? 1 : P;
#pragma unroll
        for (int l = 0; l < NF1 / P; ++l) {
            const int b = ax == 0 ? l * P : l;
#pragma unroll
            for (int q = 0; q < VB; ++q) {
                T x[P];
#pragma unroll
                for (int i = 0; i < P; ++i) x[i] = J[b + i * ts][q];
#pragma unroll
                for (int i = 0; i < P; ++i) {
                    T y = g.KW[i][0] * x[0];
#pragma unroll
                    for (int j = 1; j < P; ++j) y += g.KW[i][j] * x[j];
                    J[b + i * ts][q] = y;
                }
            }
        }
    }
    T kn[P];
#pragma unroll
    for (int i = 0; i < P; ++i) kn[i] = s ? g.kn[1][i] : g.kn[0][i];
#pragma unroll
    for (int t = 0; t < NF1; ++t) {
        const int b = line_base<ND, P>(d, t);
#pragma unroll
        for (int i = 0; i < P; ++i)
#pragma unroll
            for (int q = 0; q < VB; ++q) R[b + i * st][q] += kn[i] * J[t][q];
    }
}

// neighbour values of face (d, s)
template <int NF1, typename T, int VB>
__device__ __forceinline__ void aff_face(int i0, int Nv, int64_t v0, const T* const* rowp, const signed char* wk,
                                         Vec<T, VB> (&ur)[NF1])
{
#pragma unroll
    for (int t = 0; t < NF1; ++t) {
        int64_t off = v0;
        const int kd = wk[i0 + t];
        if (kd >= BDGFS_BC_SPECULAR_X) off = mirror_chunk(v0, Nv, kd, VB);
        ur[t].load(rowp[i0 + t] + off);
    }
}

template <typename T, int ND, int P, int VB, int OCC>
__global__ void __launch_bounds__(128, OCC) affine_kernel(const AffArgs<T, ND, P> g)
{
    constexpr int NF1 = AffShape<ND, P>::NF1, NU = AffShape<ND, P>::NU, NF = AffShape<ND, P>::NF;
    __shared__ const T* rowp[NF];          // neighbour row (or wall row, or own row to mirror) at velocity 0
    __shared__ T wsc[NF], wu[NF][3];       // wall: scale of f_w, velocity U
    __shared__ signed char wk[NF];         // boundary kind, -1 inside
    const int64_t e = blockIdx.y, nv = g.el.nv;
    for (int i = threadIdx.x; i < NF; i += blockDim.x) {
        // table entries clamped into range (a malformed table gives wrong values,
        // never an out-of-range access)
        const int f = min(max(g.fid[i], 0), NF - 1);
        const int n = g.el.nbr[e * NF + f];
        const T* own = g.uf ? g.uf + (e * NF + f) * nv : g.u + (e * NU + min(max(g.fsel[f], 0), NU - 1)) * nv;
        const T* p = own;
        int kind = -1;
        if (n >= 0) {
            if (g.uf) {
                p = g.uf + int64_t(n) * nv;
            } else if (n / NF < g.el.neles) {
                p = g.u + (int64_t(n / NF) * NU + min(max(g.fsel[n % NF], 0), NU - 1)) * nv;
            }                                          // else outside this state: no flux
        } else {
            const int w = -1 - n, bid = g.wl.bcid[w];
            kind = g.wl.kind ? g.wl.kind[bid] : BDGFS_BC_DIFFUSE;
            if (kind < BDGFS_BC_OUTLET) {
                p = static_cast<const T*>(g.wl.fw) + int64_t(bid) * nv;
                const T* bcv = static_cast<const T*>(g.wl.bcv) + 2 * w;
                wsc[i] = kind == BDGFS_BC_DIFFUSE ? -bcv[0] / bcv[1] : T(1);
                for (int k = 0; k < 3; ++k) wu[i][k] = static_cast<const T*>(g.wl.uwall)[bid * 3 + k];
            }
        }
        rowp[i] = p;
        wk[i] = static_cast<signed char>(kind);
    }
    __syncthreads();
    T S[ND][ND];
#pragma unroll
    for (int d = 0; d < ND; ++d)
#pragma unroll
        for (int k = 0; k < ND; ++k) S[d][k] = g.smat[(e * ND + d) * ND + k];
    const T rj = static_cast<const T*>(g.el.rcpdjac)[e * NU];
    const T* c0 = static_cast<const T*>(g.el.c0);
    const T* ue = g.u + e * NU * nv;
    const int64_t v1 = min((int64_t(blockIdx.x) + 1) * g.chunk, nv);
    for (int64_t v0 = int64_t(blockIdx.x) * g.chunk + int64_t(threadIdx.x) * VB; v0 < v1; v0 += 128 * VB) {
        Vec<T, VB> u[NU];
#pragma unroll
        for (int i = 0; i < NU; ++i) u[i].load(ue + i * nv + v0);
        T c[VB][3];
#pragma unroll
        for (int q = 0; q < VB; ++q) vel(c0, g.el.Nv, v0 + q, c[q]);
        T al[ND][VB];
        int sides[ND];                     // bit 0: lower face is inflow for a velocity, bit 1: upper
#pragma unroll
        for (int d = 0; d < ND; ++d) {
            sides[d] = 0;
#pragma unroll
            for (int q = 0; q < VB; ++q) {
                al[d][q] = T(0);
#pragma unroll
                for (int k = 0; k < ND; ++k) al[d][q] += S[d][k] * c[q][k];
                if (al[d][q] > T(0)) sides[d] |= 1;
                if (al[d][q] < T(0)) sides[d] |= 2;
            }
        }
        T R[NU][VB];
        // the inflow face of most chunks; a chunk with velocities of both signs
        // takes the upper face after the lower one
        const int f0 = sides[0] == 2, f1 = sides[1] == 2, f2 = ND == 3 && sides[ND - 1] == 2;
#define FACE(d, s, x) aff_face<NF1>((2 * (d) + (s)) * NF1, g.el.Nv, v0, rowp, wk, x)
#define LIFT(d, s, x) aff_lift<d>(g, S, c, s, wk, wsc, wu, x, u, al[d], R)
#define BOTH(d)                     \
    if (sides[d] == 3) {            \
        Vec<T, VB> x[NF1];          \
        FACE(d, 1, x);              \
        LIFT(d, 1, x);              \
    }
        Vec<T, VB> ua[NF1], ub[NF1];
        FACE(0, f0, ua);
        aff_volume<0>(g, u, al[0], R);
        FACE(1, f1, ub);
        LIFT(0, f0, ua);
        BOTH(0)
        aff_volume<1>(g, u, al[1], R);
        if constexpr (ND == 3) FACE(2, f2, ua);
        LIFT(1, f1, ub);
        BOTH(1)
        if constexpr (ND == 3) {
            aff_volume<2>(g, u, al[2], R);
            LIFT(2, f2, ua);
            BOTH(2)
        }
#undef FACE
#undef LIFT
#undef BOTH
        // out = a u + b L(u) + c1 x1 + c2 x2: the rows of x1, then of x2, all in
        // flight together in u's registers, and the stores last (out may be one
        // of them)
        const T br = -g.b * rj;
#pragma unroll
        for (int i = 0; i < NU; ++i)
#pragma unroll
            for (int q = 0; q < VB; ++q) R[i][q] = g.a * u[i].v[q] + br * R[i][q];
        auto add = [&](const T* x, T w) {
#pragma unroll
            for (int i = 0; i < NU; ++i) u[i].load(x + (e * NU + i) * nv + v0);
#pragma unroll
            for (int i = 0; i < NU; ++i)
#pragma unroll
                for (int q = 0; q < VB; ++q) R[i][q] += w * u[i].v[q];
        };
        if (g.x1) add(g.x1, g.c1);
        if (g.x2) add(g.x2, g.c2);
#pragma unroll
        for (int i = 0; i < NU; ++i) {
            Vec<T, VB> o;
#pragma unroll
            for (int q = 0; q < VB; ++q) o.v[q] = R[i][q];
            o.store(g.out + (e * NU + i) * nv + v0);
        }
    }
}

template <typename T, int ND, int P, int VB, int OCC = 4>
static int affine_launch_vb(const bdgfs_fr_eles& el, const bdgfs_fr_walls* wl, const bdgfs_fr_affine& af, const void* u,
                            const void* uf, void* out, double a, double b, const void* x1, double c1, const void* x2,
                            double c2, cudaStream_t st)
{
    AffArgs<T, ND, P> g{};
    g.el = el;
    if (wl) g.wl = *wl;
    g.u = static_cast<const T*>(u);
    g.uf = static_cast<const T*>(uf);
    g.fsel = af.fsel;
    g.fid = af.fid;
    g.smat = static_cast<const T*>(af.smat);
    g.out = static_cast<T*>(out);
    g.x1 = static_cast<const T*>(x1);
    g.x2 = static_cast<const T*>(x2);
    g.a = T(a);
    g.b = T(b);
    g.c1 = T(c1);
    g.c2 = T(c2);
    for (int i = 0; i < P; ++i) {
        for (int j = 0; j < P; ++j) {
            g.D[i][j] = T(af.d[i * P + j]);
            g.KW[i][j] = T(af.kw[i * P + j]);
        }
        g.kn[0][i] = T(af.kn[i]);
        g.kn[1][i] = T(af.kn[P + i]);
    }
    // steps of 128 VB velocities per CTA: several, to amortise the face table,
    // as long as the launch keeps about eight CTAs per resident one
    const int64_t step = 128 * int64_t(VB), nstep = (el.nv + step - 1) / step;
    int64_t per = std::min<int64_t>(8, nstep * el.neles / (148 * 3 * 8));
    if (per < 1) per = 1;
    while ((nstep + per - 1) / per > 65535) per *= 2;
    if (el.neles > 65535) return BDGFS_EINVAL;
    g.chunk = per * step;
    const dim3 grid(unsigned((nstep + per - 1) / per), unsigned(el.neles));
    affine_kernel<T, ND, P, VB, OCC><<<grid, 128, 0, st>>>(g);
    return cuda_status(cudaGetLastError());
}

template <typename T, int ND, int P>
static int affine_launch(const bdgfs_fr_eles& el, const bdgfs_fr_walls* wl, const bdgfs_fr_affine& af, const void* u,
                         const void* uf, void* out, double a, double b, const void* x1, double c1, const void* x2,
                         double c2, cudaStream_t st)
{
    // velocities per thread and CTAs per SM, by what a point count leaves in
    // registers; measured with three combination rows on one B200 (us, FP32):
    //   hex P2 (27 points, 210 elements, 24^3)   1 x 4: 344, 2 x 3: 465, 2 x 2: 466, 1 x 5: 633
    //   quad P3 (16, 128 elements, 24^3)         2 x 4: 86, 4 x 3: 94, 2 x 3: 97, 1 x 4: 128
    //   quad P2 (9, 35 elements, 24^3)           4 x 4: 13.8, 2 x 5: 14.6, 4 x 3: 16.7, 2 x 4: 16.7
    //   hex P1 (8, 210 elements, 24^3)           4 x 4: 94, 4 x 3: 101, 2 x 4: 108
    // and FP64 on 16^3: hex P2 1 x 3, quad P3 2 x 2, quad P2 2 x 3, others 2 x 4
    constexpr int NU = AffShape<ND, P>::NU;
    constexpr bool S = sizeof(T) == 4;
    constexpr int VB = S ? (NU > 16 ? 1 : NU > 9 ? 2 : 4) : (NU > 16 ? 1 : 2);
    constexpr int OCC = S ? 4 : (NU > 16 ? 3 : NU > 9 ? 2 : NU == 9 ? 3 : 4);
    const void* ptrs[] = {u, uf, out, x1, x2, wl ? wl->fw : nullptr};
    const int ymask = (1 << BDGFS_BC_SPECULAR_Y) | (1 << BDGFS_BC_SPECULAR_Z);
    const bool mirror_ok = !(wl && wl->kind && (wl->kinds_used & ymask)) || el.Nv % VB == 0;
    if (VB > 1 && mirror_ok && vec_width<T>(el.nv, ptrs, 6, VB) == VB)
        return affine_launch_vb<T, ND, P, VB, OCC>(el, wl, af, u, uf, out, a, b, x1, c1, x2, c2, st);
    return affine_launch_vb<T, ND, P, 1, S ? 4 : 3>(el, wl, af, u, uf, out, a, b, x1, c1, x2, c2, st);
}

}  // namespace bdgfs

using namespace bdgfs;

extern "C" int32_t bdgfs_fr_rhs_affine(const bdgfs_fr_eles* el, const bdgfs_fr_walls* wl, const bdgfs_fr_affine* af,
                                       const void* u, const void* uf, void* out, double a, double b, const void* x1,
                                       double c1, const void* x2, double c2, void* stream)
{
    if (!el || !af || el->nv < 1 || el->neles < 1 || el->Nv < 1 || el->Nv > 1024 ||
        int64_t(el->Nv) * el->Nv * el->Nv != el->nv || !el->rcpdjac || !el->nbr || !el->c0 || !af->fsel || !af->fid ||
        !af->smat || !u || !out || (!uf && out == u))
        return BDGFS_EINVAL;
    if (wl && wl->nwall > 0 && (!wl->bcid || !wl->uwall || !wl->fw || !wl->bcv)) return BDGFS_EINVAL;
    cudaStream_t st = static_cast<cudaStream_t>(stream);
#define GO(D, P, U, F)                                                                                         \
    if (el->ndims == D && af->p == P && el->nupts == U && el->nfpts == F)                                      \
        return el->fp64 ? affine_launch<double, D, P>(*el, wl, *af, u, uf, out, a, b, x1, c1, x2, c2, st)      \
                        : affine_launch<float, D, P>(*el, wl, *af, u, uf, out, a, b, x1, c1, x2, c2, st);
    GO(2, 2, 4, 8) GO(2, 3, 9, 12) GO(2, 4, 16, 16) GO(3, 2, 8, 24) GO(3, 3, 27, 54)
#undef GO
    return BDGFS_EUNSUPPORTED;
}
