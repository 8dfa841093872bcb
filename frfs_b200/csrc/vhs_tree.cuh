// Collision operator by axis-wise shifts (Nv = 24, FP32): included by
// vhs_collide.cu, whose header states the algorithm's quantities.
//
// With F = FFT(f)/n and E_pq(l) = exp(i a_pq(l)), S_p = sum_q f+ f-, where
// f+- = IFFT(E+- F) is f moved by +-(one direction's shift): the transform of
// the multiplier m_pq in vhs_collide.cu is Re(w^2) = f+ f-.  E is a product of
// one factor per axis, so a shift is three 1-D shifts, and directions with
// equal components share them: the directions form a tree whose x-nodes are
// the distinct |s_x| (a direction and its opposite give the same f+ f-),
// y-nodes the distinct s_y below an x-node and leaves the distinct |s_z| below
// a y-node, with s_z, -s_z or both.  The 12 directions of the octahedral orbit
// are 2 x-nodes, 6 y-nodes and 6 leaves with both signs.
//
// A node holds the pair (A, B) of f moved by the node's shift and by its
// opposite, one f32x2 lane each, with the axes not yet visited in spectral
// space:
//   x-node  A(x; ky, kz) = IFFT_x(E_x F),  B with conj E_x;  kz <= N/2 only
//           (A and B are transforms of real functions)
//   y-node  A(x, y; kz) = IFFT_y(E_y A),  B with conj E_y
//   leaf    w = IFFT_z((cos + sin)(kz shift) A), which is A_c - i A_s for the
//           even and odd parts A(z +- shift) = A_c +- A_s, likewise for B; then
//           A(z + g) B(z - g) + A(z - g) B(z + g) = 2 Re(w_A w_B)
//           A(z + g) B(z - g) = Re(w_A w_B) + Im(conj(w_A) w_B).
// Nyquist planes: the Hermitian part of E is Re of the product of the Nyquist
// axes' factors times the others.  Each axis carries Re E at its Nyquist index
// c; the products of two imaginary parts s s' that this leaves out on the
// Nyquist edges enter in the y-pass: at ky = N/2, -s_x s_y (-1)^x F(N/2, N/2, kz);
// the z axis needs, on the (real) plane kz = N/2, the field that its s_z
// multiplies; it rides in the imaginary part of that plane.  The result equals
// the multiplier form exactly, in exact arithmetic.
//
// Work per radius at 12 directions: 2 + 6 passes of 312 pencil pairs and one of
// 6 x 576, against 36 passes of 288 pairs, and 8 exchanges of a 120 KB cube
// through shared memory against 24 of 110 KB.  Measured on one B200, Nrho = 12,
// 12 directions: 2048 distributions 9.79 -> 5.98 ms (the variant with spectra
// in tensor memory -> this one), 97 0.705 -> 0.350 ms, one 0.706 -> 0.084 ms
// (radii cut over CTAs, split.cuh; so is the last, partly filled round of a long
// list: 1.3 % of the 2048); the error against 64-bit arithmetic falls from 4.5e-5
// to 1e-5 of Q (fewer roundings into S_p).  Bound: the FP32 pipe (51 % busy) and
// the barriers of the exchanges, at 10 warps (shared memory 44 %).
//
// One CTA of 320 threads per distribution.  Thread t < 312 owns the pencil
// (i, kz) = (t % 24, t / 24): ky in the x-passes, x in the y-passes.  Leaves:
// thread t owns the z-pencils t and t + 320 (of 576, x fastest).  Exchange
// elements are (A.re, B.re, A.im, B.im): one 16-byte access each, free of bank conflicts (row pitch 313 where the pencil axis
// changes, 312 else).  F lives in shared memory; the x-node's pencils and S_p in
// tensor memory, where only their own thread reads them (10 warps put three on
// two of the SM's sub-partitions, which caps registers at 168); the spectral
// gain G^ in global scratch (L2), touched once per radius.
#pragma once
#include "split.cuh"

namespace bdgfs {

namespace tree {
constexpr int N = 24, H = N / 2, HP = H + 1;
constexpr int NT = 320;                       // 10 warps
constexpr int NP = N * HP;                    // x / y pencils: 312
constexpr int PX = NP + 1;                    // pitch of the x -> y exchange
constexpr int NZ = N * N;                     // z pencils: 576
constexpr int kMaxM = 48;                     // directions (node tables in shared memory)
constexpr int kGroups = (NT / 32 + 3) / 4;    // TMEM column groups
constexpr uint32_t kAB = 0, kS = 4 * N * kGroups;   // TMEM columns: node pencils, S_p
constexpr uint32_t kCols = 512;
static_assert(NT >= NP && 2 * NT >= NZ && NT < NZ, "thread roles");
static_assert(kS + 2 * N * kGroups <= kCols, "TMEM columns");
}  // namespace tree

struct TreePlan {
    int nx, ny, nl;
    // node: direction | conjugate << 8; children of x-node i: y-nodes
    // xend[i-1]..xend[i)-1, of y-node j: leaves yend[j-1]..yend[j)-1
    uint16_t x[tree::kMaxM], y[tree::kMaxM], z[tree::kMaxM];
    uint8_t xend[tree::kMaxM], yend[tree::kMaxM], wp[tree::kMaxM], wm[tree::kMaxM];
};

struct QLayoutTree {
    static size_t smem_bytes(int M)
    {
        size_t b = size_t(tree::N) * tree::PX * sizeof(float4);                  // exchange
        b += size_t(tree::N) * tree::NP * sizeof(float2);                        // F
        b += size_t(M) * (2 * tree::N + tree::HP) * sizeof(float4);              // node factors
        b += size_t(M) * 2 * sizeof(float);                                      // Nyquist sines
        b += 10 * (tree::NT / 32) * sizeof(double) + 16;
        return b;
    }
    // G^ of one CTA, or of one work item when distributions are split over radii
    static constexpr size_t slot_bytes() { return size_t(tree::N) * tree::NT * sizeof(float2); }
    // per CTA: its slot, and eight for the radii of cut distributions
    static constexpr int kCut = 8;
    static size_t scratch_bytes() { return (1 + kCut) * (slot_bytes() + 256); }
};

struct TreeArgs {
    bdgfs_vhs_grid g;
    bdgfs_vhs_batch batches[4];
    int32_t nbatch, flags;
    unsigned char* slots;
    uint32_t* tickets;              // one per cut distribution, zeroed before the launch
    SplitArgs split;                // slots: radii of cut distributions, after one per CTA
    unsigned long long* counter;
};

// The direction tree, from the factors exp(i beta_p s_d) (wave number 1) of
// the first and the last radius: equal (or conjugate) values in both are equal
// (or opposite) components.  One thread.
__device__ inline void tree_plan(const cpx<float>* phase, int Nrho, int M, TreePlan& P, float4* e)
{
    using namespace tree;
    // e[q*3 + d] = factors of the first and last radius, direction flipped so
    // that its first nonzero component is positive
    auto conj4 = [](float4 v) { return make_float4(v.x, -v.y, v.z, -v.w); };
    auto same = [](float4 a, float4 b) { return a.x == b.x && a.y == b.y && a.z == b.z && a.w == b.w; };
    P.nx = P.ny = P.nl = 0;
    uint64_t used = 0;
    uint64_t flip = 0;
    for (int q = 0; q < M; ++q) {
        bool neg = false;
        for (int d = 0; d < 3; ++d) {
            const float s = e[q * 3 + d].y;
            if (s != 0.f) { neg = s < 0.f; break; }
        }
        if (neg) {
            flip |= 1ull << q;
            for (int d = 0; d < 3; ++d) e[q * 3 + d] = conj4(e[q * 3 + d]);
        }
    }
    for (int q = 0; q < M; ++q) {
        if (used >> q & 1) continue;
        P.x[P.nx] = uint16_t(q | ((flip >> q & 1) << 8));
        for (int r = q; r < M; ++r) {                        // y-nodes below x-node q
            if ((used >> r & 1) || !same(e[q * 3], e[r * 3])) continue;
            P.y[P.ny] = uint16_t(r | ((flip >> r & 1) << 8));
            for (int t = r; t < M; ++t) {                    // leaves below y-node r
                if ((used >> t & 1) || !same(e[q * 3], e[t * 3]) || !same(e[r * 3 + 1], e[t * 3 + 1])) continue;
                int wp = 0, wm = 0;
                for (int u = t; u < M; ++u) {
                    if ((used >> u & 1) || !same(e[q * 3], e[u * 3]) || !same(e[r * 3 + 1], e[u * 3 + 1])) continue;
                    if (same(e[t * 3 + 2], e[u * 3 + 2])) ++wp;
                    else if (same(e[t * 3 + 2], conj4(e[u * 3 + 2]))) ++wm;
                    else continue;
                    if (u != t) used |= 1ull << u;
                }
                used |= 1ull << t;
                P.z[P.nl] = uint16_t(t | ((flip >> t & 1) << 8));
                P.wp[P.nl] = uint8_t(wp);
                P.wm[P.nl] = uint8_t(wm);
                ++P.nl;
            }
            P.yend[P.ny++] = uint8_t(P.nl);
        }
        P.xend[P.nx++] = uint8_t(P.ny);
    }
}

__global__ void __launch_bounds__(tree::NT, 1) vhs_tree_kernel(const TreeArgs a)
{
    using namespace tree;
    extern __shared__ __align__(16) unsigned char smem[];
    __shared__ int64_t s_item;
    __shared__ int64_t s_start[5];
    __shared__ SplitPlan s_plan;
    __shared__ int s_last;
    __shared__ volatile int s_lost;
    __shared__ uint32_t s_tmem;
    __shared__ __align__(8) uint64_t s_free;
    __shared__ TreePlan pl;

    const bdgfs_vhs_grid& g = a.g;
    const int tid = threadIdx.x, warp = tid >> 5, M = g.M, Nrho = g.Nrho;
    float4* buf = reinterpret_cast<float4*>(smem);
    float2* buf2 = reinterpret_cast<float2*>(smem);
    float2* Fs = reinterpret_cast<float2*>(buf + N * PX);          // [kx][t]
    float4* xt = reinterpret_cast<float4*>(Fs + N * NP);           // [node][k]: (c, c, s, -s)
    float4* yt = xt + M * N;
    float4* zt = yt + M * N;                                       // [leaf][k <= H]: (m+, m+, m-, m-)
    float* xs = reinterpret_cast<float*>(zt + M * HP);             // Nyquist sines
    float* ys = xs + M;
    double* red = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(ys + M) + 15) & ~uintptr_t(15));

    const cpx<float>* phase = static_cast<const cpx<float>*>(g.phase);
    const float* gw = static_cast<const float*>(g.gw);
    const float* bb2 = static_cast<const float*>(g.bb2);
    const int project = a.flags & BDGFS_PROJECT;

    if (tid == 0) {
        tc::mbar_init(&s_free, NT);
        s_lost = 0;
    }
    for (int i = tid; i < 3 * M; i += NT) {
        const cpx<float> v = phase[i * N + 1], w = phase[size_t(Nrho - 1) * M * 3 * N + i * N + 1];
        buf[i] = make_float4(v.x, v.y, w.x, w.y);
    }
    if (tid == 32) {
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
    // nothing to do (a device count of zero): leave before the tree and tensor memory
    // (18.5 -> 7.3 us with the launch's two memsets, one B200)
    if (s_start[a.nbatch] == 0) return;
    if (tid < 32) tc::tmem_alloc(&s_tmem, kCols);
    tc::tc_fence_before();
    if (tid == 32) tree_plan(phase, Nrho, M, pl, buf);
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t lane0 = s_tmem + (uint32_t(32 * (warp & 3)) << 16);
    const uint32_t tab = lane0 + kAB + uint32_t(4 * N * (warp >> 2));
    const uint32_t tsp = lane0 + kS + uint32_t(2 * N * (warp >> 2));     // S_p of z-pencil 0; + N: of 1

    // pencil (i, kz) of the x- and y-passes; threads 312.. repeat the last one
    // (tensor-memory accesses are warp-wide) and store nothing
    const int te = tid < NP ? tid : NP - 1;
    const bool on = tid < NP;
    const int kz = te / N, pi = te - kz * N;
    const float alt = (pi & 1) ? -1.f : 1.f;             // (-1)^x in the y-passes
    const int z0 = (tid / N) * NP + tid % N;             // z-pencil tid: y * NP + x (+ kz * N)
    const int z1 = ((tid + NT) / N) * NP + (tid + NT) % N;
    const bool two = tid + NT < NZ;

    // Exchange round: wait until every thread has read the last one's
    // elements, store, barrier, load, arrive.  The wait is bounded; on expiry the
    // CTA gives NaN.
    uint32_t par = 1;
    auto wait_free = [&]() {
        tc::mbar_wait_or_lose(&s_free, par, &s_lost);
        par ^= 1u;
        __syncwarp();
    };
    auto arrive = [&]() { tc::mbar_arrive(&s_free); };

    // (re, im) *= (c + i s) on lane A and (c - i s) on lane B
    auto rot = [](float4 e, float2& re, float2& im) {
        const float2 C = f2(e.x, e.y), S = f2(e.z, e.w), nS = f2(e.w, e.z);
        const float2 r = __ffma2_rn(im, nS, __fmul2_rn(re, C));
        im = __ffma2_rn(re, S, __fmul2_rn(im, C));
        re = r;
    };
    auto put = [&](int pitch, const float2 (&vr)[N], const float2 (&vi)[N]) {
        if (on) {
#pragma unroll
            for (int k = 0; k < N; ++k) buf[k * pitch + te] = make_float4(vr[k].x, vr[k].y, vi[k].x, vi[k].y);
        }
    };
    // y-pencil of an x -> y exchange
    auto get_y = [&](float2 (&vr)[N], float2 (&vi)[N]) {
        const float4* b = buf + pi * PX + kz * N;
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float4 v = b[k];
            vr[k] = f2(v.x, v.y);
            vi[k] = f2(v.z, v.w);
        }
    };
    // forward 3-D transform of the real cube whose z-pencils tid and tid + NT
    // are u0, u1: twice the spectrum X[kx] at this thread's (ky, kz)
    auto forward = [&](const float (&u0)[N], const float (&u1)[N], cpx<float> (&X)[N]) {
#pragma unroll
        for (int z = 0; z < N; ++z) X[z] = {u0[z], u1[z]};
        dft<N, -1>(X);
        wait_free();
#pragma unroll
        for (int k = 0; k <= H; ++k) {
            const cpx<float> p = X[k], m = X[(N - k) % N];
            buf2[z0 + k * N] = f2(p.x + m.x, p.y - m.y);
            if (two) buf2[z1 + k * N] = f2(p.y + m.y, m.x - p.x);
        }
        __syncthreads();
#pragma unroll
        for (int y = 0; y < N; ++y) {
            const float2 v = buf2[y * NP + te];
            X[y] = {v.x, v.y};
        }
        arrive();
        dft<N, -1>(X);
        wait_free();
        if (on) {
#pragma unroll
            for (int k = 0; k < N; ++k) buf2[pi * PX + kz * N + k] = f2(X[k].x, X[k].y);
        }
        __syncthreads();
#pragma unroll
        for (int x = 0; x < N; ++x) {
            const float2 v = buf2[x * PX + te];
            X[x] = {v.x, v.y};
        }
        arrive();
        dft<N, -1>(X);
    };
    auto load_row = [&](const float* p, bool vec, float (&u)[N]) {
        if (vec) {
#pragma unroll
            for (int z = 0; z < N; z += 4) {
                const float4 v = *reinterpret_cast<const float4*>(p + z);
                u[z] = v.x; u[z + 1] = v.y; u[z + 2] = v.z; u[z + 3] = v.w;
            }
        } else {
#pragma unroll
            for (int z = 0; z < N; ++z) u[z] = p[z];
        }
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
        if (dof < 0 || dof >= bt.ndof) continue;           // malformed index list: skip
        constexpr int n3 = N * N * N;
        const float* f = static_cast<const float*>(bt.f) + dof * n3;
        const bool fvec = (reinterpret_cast<uintptr_t>(f) & 15u) == 0;
        // row (x, y) of z-pencil j = y N + x
        const int row0 = ((tid % N) * N + tid / N) * N;
        const int row1 = two ? (((tid + NT) % N) * N + (tid + NT) / N) * N : row0;

        // ---- F = FFT(f) / n ----
        {
            float u0[N], u1[N];
            load_row(f + row0, fvec, u0);
            load_row(f + row1, fvec, u1);
            cpx<float> X[N];
            forward(u0, u1, X);
            const float sc = 0.5f / float(n3);
            if (on) {
#pragma unroll
                for (int k = 0; k < N; ++k) Fs[k * NP + te] = f2(X[k].x * sc, X[k].y * sc);
            }
        }

        // G^ of this thread, [kx * NT]: the sum so far, or one slot per radius (cut)
        const int64_t slot = ns > 1 ? a.split.nctas + it.cut * Nrho + it.b0 : int64_t(blockIdx.x);
        float2* G = reinterpret_cast<float2*>(a.slots + size_t(slot) * QLayoutTree::slot_bytes()) + tid;
        for (int p = it.b0; p < it.b1; ++p) {
            // ---- node factors of radius p ----
            const cpx<float>* php = phase + size_t(p) * M * 3 * N;
            for (int i = tid; i < (pl.nx + pl.ny) * N; i += NT) {
                const bool isx = i < pl.nx * N;
                const int j = isx ? i : i - pl.nx * N;
                const int node = j / N, k = j - node * N;
                const int w = isx ? pl.x[node] : pl.y[node];
                cpx<float> v = php[((w & 255) * 3 + (isx ? 0 : 1)) * N + k];
                if (w >> 8) v.y = -v.y;
                if (k == H) {
                    (isx ? xs : ys)[node] = v.y;
                    v.y = 0.f;
                }
                (isx ? xt : yt)[j] = make_float4(v.x, v.x, v.y, -v.y);
            }
            for (int i = tid; i < pl.nl * HP; i += NT) {
                const int leaf = i / HP, k = i - leaf * HP, w = pl.z[leaf];
                cpx<float> v = php[((w & 255) * 3 + 2) * N + k];
                if (w >> 8) v.y = -v.y;
                const float m = v.x + v.y, mm = v.x - v.y;
                zt[i] = k == H ? make_float4(v.x, v.x, v.y, v.y) : make_float4(m, m, mm, mm);
            }
            __syncthreads();                               // factors (and F) in place

            {
                uint32_t r[16];
#pragma unroll
                for (int k = 0; k < 16; ++k) r[k] = 0u;
#pragma unroll
                for (int c = 0; c < 2 * N / 16; ++c) tc::tmem_st16(tsp + 16 * c, r);
                tc::tmem_wait_st();
            }
            int yn = 0;
#pragma unroll 1
            for (int xn = 0; xn < pl.nx; ++xn) {
                const float sx = xs[xn];
                {
                    float2 vr[N], vi[N];
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        const float2 F = Fs[k * NP + te];
                        vr[k] = f2(F.x, F.x);
                        vi[k] = f2(F.y, F.y);
                        rot(xt[xn * N + k], vr[k], vi[k]);
                    }
                    dft_p2<N, +1>(vr, vi);
                    wait_free();
                    put(PX, vr, vi);
                    __syncthreads();
                    get_y(vr, vi);
                    arrive();
#pragma unroll
                    for (int c = 0; c < N / 4; ++c) {
                        uint32_t r[16];
#pragma unroll
                        for (int k = 0; k < 4; ++k) {
                            r[4 * k] = __float_as_uint(vr[4 * c + k].x);
                            r[4 * k + 1] = __float_as_uint(vr[4 * c + k].y);
                            r[4 * k + 2] = __float_as_uint(vi[4 * c + k].x);
                            r[4 * k + 3] = __float_as_uint(vi[4 * c + k].y);
                        }
                        tc::tmem_st16(tab + 16 * c, r);
                    }
                    tc::tmem_wait_st();
                }
#pragma unroll 1
                for (; yn < pl.xend[xn]; ++yn) {
                    {
                        const float sy = ys[yn];
                        const float4* e = yt + yn * N;
                        float2 vr[N], vi[N];
                        float2 nr, ni;                      // the node's pencil at ky = N/2, before the shift
#pragma unroll
                        for (int c = 0; c < N / 4; ++c) {
                            uint32_t r[16];
                            tc::tmem_ld16_issue(tab + 16 * c, r);
                            tc::tmem_wait();
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                const int kk = 4 * c + k;
                                vr[kk] = f2(__uint_as_float(r[4 * k]), __uint_as_float(r[4 * k + 1]));
                                vi[kk] = f2(__uint_as_float(r[4 * k + 2]), __uint_as_float(r[4 * k + 3]));
                                if (kk == H) { nr = vr[kk]; ni = vi[kk]; }
                                rot(e[kk], vr[kk], vi[kk]);
                            }
                        }
                        {
                            const float2 F = Fs[H * NP + kz * N + H];
                            const float w = -alt * sx * sy;
                            vr[H].x += w * F.x; vr[H].y += w * F.x;
                            vi[H].x += w * F.y; vi[H].y += w * F.y;
                        }
                        if (kz == H) {                      // one warp: the field that s_z multiplies
                            const float w = alt * sx;
                            const float2 G = f2(w, -w), nG = f2(-w, w);
#pragma unroll
                            for (int k = 0; k < N; ++k) {
                                const float2 F = Fs[H * NP + H * N + k];
                                float2 pr = f2(F.x, F.x), qi = f2(F.y, F.y);
                                rot(e[k], pr, qi);
                                vr[k] = __ffma2_rn(nG, qi, vr[k]);
                                vi[k] = __ffma2_rn(G, pr, vi[k]);
                            }
                            vr[H] = __ffma2_rn(f2(-sy, sy), ni, vr[H]);
                            vi[H] = __ffma2_rn(f2(sy, -sy), nr, vi[H]);
                        }
                        dft_p2<N, +1>(vr, vi);
                        wait_free();
                        put(NP, vr, vi);
                        __syncthreads();
                    }
                    const int l0 = yn ? pl.yend[yn - 1] : 0, l1 = pl.yend[yn];
#pragma unroll 1
                    for (int l = l0; l < l1; ++l) {
                        const float wr = 0.5f * float(pl.wp[l] + pl.wm[l]), wi = 0.5f * float(pl.wp[l] - pl.wm[l]);
#pragma unroll
                        for (int r = 0; r < 2; ++r) {
                            if (r && !two) {
                                if (l + 1 == l1) arrive();
                                break;
                            }
                            const float4* bz = buf + (r ? z1 : z0);
                            float2 vr[N], vi[N];
                            const float4* e = zt + l * HP;
#pragma unroll
                            for (int k = 0; k <= H; ++k) {
                                const float4 v = bz[k * N];
                                const float2 re = f2(v.x, v.y), im = f2(v.z, v.w);
                                if (k == 0) {
                                    vr[0] = re;
                                    vi[0] = im;
                                } else if (k == H) {
                                    vr[k] = __fmul2_rn(re, f2(e[k].x, e[k].y));
                                    vi[k] = __fmul2_rn(im, f2(e[k].z, e[k].w));
                                } else {
                                    const float4 m = e[k];
                                    vr[k] = __fmul2_rn(re, f2(m.x, m.y));
                                    vi[k] = __fmul2_rn(im, f2(m.x, m.y));
                                    vr[N - k] = __fmul2_rn(re, f2(m.z, m.w));
                                    vi[N - k] = __fmul2_rn(im, f2(-m.z, -m.w));
                                }
                            }
                            if (r && l + 1 == l1) arrive();
                            dft_p2<N, +1>(vr, vi);
                            const bool pair = wr == 1.f && wi == 0.f;
                            tc::tmem_wait_st();
#pragma unroll
                            for (int c = 0; c < N / 8; ++c) {
                                uint32_t s[8];
                                tc::tmem_ld8_issue(tsp + r * N + 8 * c, s);
                                tc::tmem_wait();
#pragma unroll
                                for (int k = 0; k < 8; ++k) {
                                    const int z = 8 * c + k;
                                    const float re = fmaf(vr[z].x, vr[z].y, -vi[z].x * vi[z].y);
                                    float v = __uint_as_float(s[k]);
                                    if (pair) {
                                        v += re;
                                    } else {
                                        const float im = vr[z].x * vi[z].y - vi[z].x * vr[z].y;
                                        v = fmaf(wr, re, fmaf(wi, im, v));
                                    }
                                    s[k] = __float_as_uint(v);
                                }
                                tc::tmem_st8(tsp + r * N + 8 * c, s);
                            }
                        }
                    }
                }
            }

            // ---- G^ += gw_p FFT(S_p); S is half the sum, forward() doubles it ----
            {
                float u0[N], u1[N];
                tc::tmem_wait_st();
#pragma unroll
                for (int c = 0; c < N / 8; ++c) {
                    uint32_t r[8], q[8];
                    tc::tmem_ld8_issue(tsp + 8 * c, r);
                    tc::tmem_ld8_issue(tsp + N + 8 * c, q);
                    tc::tmem_wait();
#pragma unroll
                    for (int k = 0; k < 8; ++k) {
                        u0[8 * c + k] = __uint_as_float(r[k]);
                        u1[8 * c + k] = __uint_as_float(q[k]);
                    }
                }
                cpx<float> X[N];
                forward(u0, u1, X);
                const float* gwp = gw + (size_t(p) * N + kz) * HP * N + pi;
                const bool acc = ns == 1 && p > 0;
#pragma unroll
                for (int kx = 0; kx < N; ++kx) {
                    const float w = ldg(gwp + (kx <= H ? kx : N - kx) * N);
                    const float2 o = acc ? G[kx * NT] : f2(0.f, 0.f);
                    G[kx * NT] = f2(__fadd_rn(o.x, __fmul_rn(w, X[kx].x)), __fadd_rn(o.y, __fmul_rn(w, X[kx].y)));
                }
                if (ns > 1) G += N * NT;
            }
        }

        float2 vr[N], vi[N];                              // lane A: this thread's G^
        if (ns > 1) {
            // the part that arrives last adds the radii in order and finishes the
            // distribution
            if (s_lost) G[-N * NT].x = tc::lost_nan(&s_lost, 0.f);
            __threadfence();
            __syncthreads();
            if (tid == 0) s_last = atomicAdd(a.tickets + it.cut, 1u) == uint32_t(ns - 1);
            __syncthreads();
            if (!s_last) continue;
            __threadfence();
            const float2* Gj = reinterpret_cast<const float2*>(a.slots + size_t(a.split.nctas + it.cut * Nrho) * QLayoutTree::slot_bytes()) + tid;
#pragma unroll
            for (int k = 0; k < N; ++k) vr[k].x = vi[k].x = 0.f;
#pragma unroll 1
            for (int j = 0; j < Nrho; ++j, Gj += N * NT) {
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const float2 v = __ldcg(Gj + k * NT);
                    vr[k].x = __fadd_rn(vr[k].x, v.x);
                    vi[k].x = __fadd_rn(vi[k].x, v.y);
                }
            }
        } else {
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const float2 v = G[k * NT];
                vr[k].x = v.x;
                vi[k].x = v.y;
            }
        }

        // ---- lane A: QG = IFFT(G^), lane B: fC = IFFT(bb2 F) ----
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float2 F = Fs[k * NP + te];
            const float w = ldg(bb2 + (kz * N + k) * N + pi);
            vr[k].y = w * F.x;
            vi[k].y = w * F.y;
        }
        dft_p2<N, +1>(vr, vi);
        wait_free();
        put(PX, vr, vi);
        __syncthreads();
        get_y(vr, vi);
        arrive();
        dft_p2<N, +1>(vr, vi);
        wait_free();
        put(NP, vr, vi);
        __syncthreads();
        const float prefac = float(g.prefac);
        double* mom = bt.moments ? bt.moments + dof * 10 : nullptr;
        const bool need_m = project || mom;
        float S[2][N];                                    // the z-pencils' f, then Q
        double m[5] = {0, 0, 0, 0, 0};
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (r && !two) {
                arrive();
                break;
            }
            const float4* bz = buf + (r ? z1 : z0);
#pragma unroll
            for (int k = 0; k <= H; ++k) {
                const float4 v = bz[k * N];
                vr[k] = f2(v.x, v.y);
                vi[k] = f2(v.z, v.w);
                if (k > 0 && k < H) {
                    vr[N - k] = vr[k];
                    vi[N - k] = f2(-v.z, -v.w);
                }
            }
            if (r) arrive();
            vr[0].x = tc::lost_nan(&s_lost, vr[0].x);
            dft_p2<N, +1>(vr, vi);
            load_row(f + (r ? row1 : row0), fvec, S[r]);
            double q0 = 0.0, q1 = 0.0, q2 = 0.0;
#pragma unroll
            for (int z = 0; z < N; ++z) {
                const float q = prefac * (vr[z].x - S[r][z] * vr[z].y);
                S[r][z] = q;
                if (need_m) {
                    const double cz = g.c0[z], dq = double(q);
                    q0 += dq;
                    q1 += cz * dq;
                    q2 += cz * cz * dq;
                }
            }
            if (need_m) {
                const int j = tid + r * NT;
                const double cx = g.c0[j % N], cy = g.c0[j / N];
                m[0] += q0;
                m[1] += cx * q0;
                m[2] += cy * q0;
                m[3] += q1;
                m[4] += (cx * cx + cy * cy) * q0 + q2;
            }
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
        float* Q = static_cast<float*>(bt.Q) + dof * n3;
        const bool qvec = (reinterpret_cast<uintptr_t>(Q) & 15u) == 0;
        double m2[5] = {0, 0, 0, 0, 0};
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            if (r && !two) break;
            if (project) {
                const int j = tid + r * NT;
                const double cx = g.c0[j % N], cy = g.c0[j / N];
                const double base = lam[0] + lam[1] * cx + lam[2] * cy + lam[4] * (cx * cx + cy * cy);
                double q0 = 0.0, q1 = 0.0, q2 = 0.0;
#pragma unroll
                for (int z = 0; z < N; ++z) {
                    const double cz = g.c0[z];
                    const double qc = double(S[r][z]) - (base + (lam[3] + lam[4] * cz) * cz);
                    S[r][z] = float(qc);
                    q0 += qc;
                    q1 += cz * qc;
                    q2 += cz * cz * qc;
                }
                m2[0] += q0;
                m2[1] += cx * q0;
                m2[2] += cy * q0;
                m2[3] += q1;
                m2[4] += (cx * cx + cy * cy) * q0 + q2;
            }
            float* qr = Q + (r ? row1 : row0);
            if (qvec) {
#pragma unroll
                for (int z = 0; z < N; z += 4)
                    __stcs(reinterpret_cast<float4*>(qr + z),
                           make_float4(S[r][z], S[r][z + 1], S[r][z + 2], S[r][z + 3]));
            } else {
#pragma unroll
                for (int z = 0; z < N; ++z) __stcs(qr + z, S[r][z]);
            }
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
    }
    tc::tmem_wait_st();
    tc::tc_fence_before();
    __syncthreads();
    if (tid < 32) {
        tc::tc_fence_after();
        tc::tmem_dealloc(s_tmem, kCols);
    }
}

}  // namespace bdgfs
