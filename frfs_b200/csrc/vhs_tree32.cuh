// Collision operator by axis-wise shifts at Nv = 32, FP32 (vhs_tree.cuh states
// the method, the direction tree and the node factors).
//
// The pencil of a pass is a lane: lanes are the 32 ky of the x-passes, the 32 x of
// the y- and z-passes.  Warp w owns kz = w and w + 8 (and warp 0 kz = 16) of the x-
// and y-passes and y = w, w + 8, w + 16, w + 24 of the z-passes.  So x -> y is a
// transpose inside a warp, and only y -> z crosses warps: its 278 KB (A and B, kz
// <= 16) go half through shared memory (y < 16) and half through the CTA's L2
// scratch.  The node pencils fill tensor memory (two kz of a warp: 256 columns,
// two warps per lane quarter); those of kz = 16 sit in shared memory.  F, S_p and
// G^ live in the CTA's scratch (L2), read and written by their own lanes only.
//
// 8 warps, so a thread may hold a 32-point pair (128 registers) beside what it works
// with.  Measured on one B200, Nrho = 16, 12 directions: 501 distributions 15.4 ->
// 7.87 ms (the warp-slab variant -> this one).  Bound: the latency of L2 (F, S_p and
// half of the y -> z exchange) with 8 warps to hide it; the FP32 pipe is 33 % busy.
#pragma once
#include "vhs_tree.cuh"

namespace bdgfs {

namespace tree32 {
constexpr int N = 32, H = 16, HP = 17, NT = 256, n = N * N * N;
constexpr int ROW = HP * N;                        // (kz, lane) entries of one k: 544
constexpr int PY = ROW + 1;                        // pitch of the 8-byte exchange
constexpr int TP = N + 1;                          // pitch of a warp's transpose
constexpr int kMaxM = 48;
constexpr size_t kX = size_t(N) * PY * sizeof(float2);          // exchange region: 139,520
static_assert(kX >= size_t(16) * ROW * sizeof(float4) && kX >= size_t(8) * N * TP * sizeof(float4), "exchange");
constexpr size_t kRow2 = size_t(N) * ROW * sizeof(float2);      // F, G^: 139,264
constexpr size_t kHalf = size_t(16) * ROW * sizeof(float4);     // y >= 16 of the y -> z exchange
constexpr size_t kS = size_t(n) * sizeof(float);
constexpr size_t kPriv = kRow2 + kHalf + kS;
}  // namespace tree32

struct QLayoutTree32 {
    static size_t smem_bytes(int M)
    {
        using namespace tree32;
        return kX + size_t(N) * N * sizeof(float4) + size_t(M) * (2 * N + HP) * sizeof(float4) +
               (N + HP) * sizeof(float2) + size_t(M) * 2 * sizeof(float) + 10 * (NT / 32) * sizeof(double) + 16;
    }
    static constexpr size_t slot_bytes() { return tree32::kRow2; }
    // per CTA: its private arrays, a slot, and eight for the radii of cut distributions
    static constexpr int kCut = 8;
    static size_t scratch_bytes() { return tree32::kPriv + (1 + kCut) * (slot_bytes() + 256); }
};

struct Tree32Args {
    bdgfs_vhs_grid g;
    bdgfs_vhs_batch batches[4];
    int32_t nbatch, flags;
    unsigned char* priv;
    unsigned char* slots;
    uint32_t* tickets;
    SplitArgs split;                // slots: radii of cut distributions, after one per CTA
    unsigned long long* counter;
};

__global__ void __launch_bounds__(tree32::NT, 1) vhs_tree32_kernel(const Tree32Args a)
{
    using namespace tree32;
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
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, M = g.M, Nrho = g.Nrho;
    float4* buf = reinterpret_cast<float4*>(smem);
    float2* buf2 = reinterpret_cast<float2*>(smem);
    float4* ab16 = reinterpret_cast<float4*>(smem + kX);           // node pencils of kz = 16: [k][lane]
    float4* xt = ab16 + N * N;
    float4* yt = xt + M * N;
    float4* zt = yt + M * N;
    float2* fh = reinterpret_cast<float2*>(zt + M * HP);           // F(H, k, H), k < N; F(H, H, kz)
    float* xs = reinterpret_cast<float*>(fh + N + HP);
    float* ys = xs + M;
    double* red = reinterpret_cast<double*>((reinterpret_cast<uintptr_t>(ys + M) + 15) & ~uintptr_t(15));
    float4* tr = buf + warp * N * TP;                              // the warp's transpose

    unsigned char* priv = a.priv + size_t(blockIdx.x) * kPriv;
    float2* F = reinterpret_cast<float2*>(priv) + lane;            // [kx][kz][ky]
    float4* half = reinterpret_cast<float4*>(priv + kRow2) + lane; // [y - 16][kz][x]
    float4* Sp = reinterpret_cast<float4*>(priv + kRow2 + kHalf) + lane;   // [z / 4][y][x]

    const cpx<float>* phase = static_cast<const cpx<float>*>(g.phase);
    const float* gw = static_cast<const float*>(g.gw);
    const float* bb2 = static_cast<const float*>(g.bb2);
    const int project = a.flags & BDGFS_PROJECT;
    const int ntask = warp == 0 ? 3 : 2;                           // kz of the x- and y-passes
    auto kz_of = [&](int r) { return r == 2 ? H : warp + 8 * r; };

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
    if (tid < 32) tc::tmem_alloc(&s_tmem, 512);
    tc::tc_fence_before();
    if (tid == 32) tree_plan(phase, Nrho, M, pl, buf);
    __syncthreads();
    tc::tc_fence_after();
    const uint32_t tab = s_tmem + (uint32_t(32 * (warp & 3)) << 16) + uint32_t(256 * (warp >> 2));   // + 128 r

    uint32_t par = 1;
    auto wait_free = [&]() {
        tc::mbar_wait_or_lose(&s_free, par, &s_lost);
        par ^= 1u;
        __syncwarp();
    };
    auto arrive = [&]() { tc::mbar_arrive(&s_free); };
    auto rot = [](float4 e, float2& re, float2& im) {
        const float2 C = f2(e.x, e.y), S = f2(e.z, e.w), nS = f2(e.w, e.z);
        const float2 r = __ffma2_rn(im, nS, __fmul2_rn(re, C));
        im = __ffma2_rn(re, S, __fmul2_rn(im, C));
        re = r;
    };
    // ky-lanes -> x-lanes of one kz, in the warp's transpose
    auto turn = [&](float2 (&vr)[N], float2 (&vi)[N]) {
        __syncwarp();
#pragma unroll
        for (int k = 0; k < N; ++k) tr[k * TP + lane] = make_float4(vr[k].x, vr[k].y, vi[k].x, vi[k].y);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < N; ++k) {
            const float4 v = tr[lane * TP + k];
            vr[k] = f2(v.x, v.y);
            vi[k] = f2(v.z, v.w);
        }
    };
    // y-pass result to the y -> z exchange
    auto put_z = [&](int kz, const float2 (&vr)[N], const float2 (&vi)[N]) {
#pragma unroll
        for (int y = 0; y < 16; ++y) buf[y * ROW + kz * N + lane] = make_float4(vr[y].x, vr[y].y, vi[y].x, vi[y].y);
#pragma unroll
        for (int y = 16; y < N; ++y)
            __stcg(half + (y - 16) * ROW + kz * N, make_float4(vr[y].x, vr[y].y, vi[y].x, vi[y].y));
    };
    auto get_z = [&](int j, int kz) -> float4 {                    // z-pencil j: y = warp + 8 j
        const int y = warp + 8 * j;
        return j < 2 ? buf[y * ROW + kz * N + lane] : __ldcg(half + (y - 16) * ROW + kz * N);
    };
    // forward 3-D transform of the real cube whose z-pencil y = warp + 8 j is
    // row(j, u): twice the spectrum at (ky = lane, kz) to out(kz, lane r of the
    // packed pair or the single kz = 16, X)
    auto forward_zy = [&](auto row) {
        float2 vr[N], vi[N];
        {
            float u[N];
            row(0, u);
#pragma unroll
            for (int z = 0; z < N; ++z) vr[z].x = u[z];
            row(1, u);
#pragma unroll
            for (int z = 0; z < N; ++z) vi[z].x = u[z];
            row(2, u);
#pragma unroll
            for (int z = 0; z < N; ++z) vr[z].y = u[z];
            row(3, u);
#pragma unroll
            for (int z = 0; z < N; ++z) vi[z].y = u[z];
        }
        dft_p2<N, -1>(vr, vi);
        wait_free();
#pragma unroll
        for (int k = 0; k <= H; ++k) {
            const int m = (N - k) % N;
            float2* o = buf2 + warp * PY + k * N + lane;
            o[0] = f2(vr[k].x + vr[m].x, vi[k].x - vi[m].x);
            o[8 * PY] = f2(vi[k].x + vi[m].x, vr[m].x - vr[k].x);
            o[16 * PY] = f2(vr[k].y + vr[m].y, vi[k].y - vi[m].y);
            o[24 * PY] = f2(vi[k].y + vi[m].y, vr[m].y - vr[k].y);
        }
        __syncthreads();
    };
    // y, then x (inside the warp), of kz = warp and warp + 8 as a pair
    auto forward_pair = [&](float2 (&vr)[N], float2 (&vi)[N]) {
        float2* p = buf2 + warp * N + lane;
#pragma unroll
        for (int y = 0; y < N; ++y) {
            const float2 s = p[y * PY], t = p[y * PY + 8 * N];
            vr[y] = f2(s.x, t.x);
            vi[y] = f2(s.y, t.y);
        }
        dft_p2<N, -1>(vr, vi);
#pragma unroll
        for (int y = 0; y < N; ++y) {
            p[y * PY] = f2(vr[y].x, vi[y].x);
            p[y * PY + 8 * N] = f2(vr[y].y, vi[y].y);
        }
        __syncwarp();
        const float2* q = buf2 + lane * PY + warp * N;
#pragma unroll
        for (int x = 0; x < N; ++x) {
            const float2 s = q[x], t = q[x + 8 * N];
            vr[x] = f2(s.x, t.x);
            vi[x] = f2(s.y, t.y);
        }
        dft_p2<N, -1>(vr, vi);
    };
    auto forward_16 = [&](cpx<float> (&X)[N]) {                    // kz = 16 (warp 0)
        float2* p = buf2 + H * N + lane;
#pragma unroll
        for (int y = 0; y < N; ++y) X[y] = {p[y * PY].x, p[y * PY].y};
        dft<N, -1>(X);
#pragma unroll
        for (int y = 0; y < N; ++y) p[y * PY] = f2(X[y].x, X[y].y);
        __syncwarp();
        const float2* q = buf2 + lane * PY + H * N;
#pragma unroll
        for (int x = 0; x < N; ++x) X[x] = {q[x].x, q[x].y};
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

    const SplitPlan plan = s_plan;
    const int64_t nitems = split_items(s_start[a.nbatch], plan);
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
        if (dof < 0 || dof >= bt.ndof) continue;                   // malformed index list: skip
        const float* f = static_cast<const float*>(bt.f) + dof * n;
        const bool fvec = (reinterpret_cast<uintptr_t>(f) & 15u) == 0;
        auto row_at = [&](int j) { return (lane * N + warp + 8 * j) * N; };    // z-pencil j of the thread

        // ---- F = FFT(f) / n ----
        forward_zy([&](int j, float (&u)[N]) { load_row(f + row_at(j), fvec, u); });
        {
            const float sc = 0.5f / float(n);
            float2 vr[N], vi[N];
            forward_pair(vr, vi);
#pragma unroll
            for (int k = 0; k < N; ++k) {
                F[k * ROW + warp * N] = f2(vr[k].x * sc, vi[k].x * sc);
                F[k * ROW + (warp + 8) * N] = f2(vr[k].y * sc, vi[k].y * sc);
            }
            if (lane == H) {
                fh[N + warp] = f2(vr[H].x * sc, vi[H].x * sc);
                fh[N + warp + 8] = f2(vr[H].y * sc, vi[H].y * sc);
            }
            if (warp == 0) {
                cpx<float> X[N];
                forward_16(X);
#pragma unroll
                for (int k = 0; k < N; ++k) F[k * ROW + H * N] = f2(X[k].x * sc, X[k].y * sc);
                fh[lane] = f2(X[H].x * sc, X[H].y * sc);
                if (lane == H) fh[N + H] = f2(X[H].x * sc, X[H].y * sc);
            }
            arrive();
        }

        // G^ [kx][kz][ky]: the sum so far, or one slot per radius (cut)
        const int64_t slot = ns > 1 ? a.split.nctas + it.cut * Nrho + it.b0 : int64_t(blockIdx.x);
        float2* G = reinterpret_cast<float2*>(a.slots + size_t(slot) * QLayoutTree32::slot_bytes()) + lane;
        for (int p = it.b0; p < it.b1; ++p) {
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
            __syncthreads();                                       // factors (and fh) in place

            bool first = true;                                     // S_p not yet written
            int yn = 0;
#pragma unroll 1
            for (int xn = 0; xn < pl.nx; ++xn) {
                const float sx = xs[xn];
                wait_free();
#pragma unroll 1
                for (int r = 0; r < ntask; ++r) {
                    const int kz = kz_of(r);
                    float2 vr[N], vi[N];
#pragma unroll
                    for (int k = 0; k < N; ++k) {
                        const float2 v = F[k * ROW + kz * N];
                        vr[k] = f2(v.x, v.x);
                        vi[k] = f2(v.y, v.y);
                    }
#pragma unroll
                    for (int k = 0; k < N; ++k) rot(xt[xn * N + k], vr[k], vi[k]);
                    dft_p2<N, +1>(vr, vi);
                    turn(vr, vi);
                    if (r + 1 == ntask) arrive();
                    if (r == 2) {
#pragma unroll
                        for (int k = 0; k < N; ++k) ab16[k * N + lane] = make_float4(vr[k].x, vr[k].y, vi[k].x, vi[k].y);
                    } else {
#pragma unroll
                        for (int c = 0; c < N / 4; ++c) {
                            uint32_t u[16];
#pragma unroll
                            for (int k = 0; k < 4; ++k) {
                                u[4 * k] = __float_as_uint(vr[4 * c + k].x);
                                u[4 * k + 1] = __float_as_uint(vr[4 * c + k].y);
                                u[4 * k + 2] = __float_as_uint(vi[4 * c + k].x);
                                u[4 * k + 3] = __float_as_uint(vi[4 * c + k].y);
                            }
                            tc::tmem_st16(tab + 128 * r + 16 * c, u);
                        }
                    }
                }
                tc::tmem_wait_st();
#pragma unroll 1
                for (; yn < pl.xend[xn]; ++yn) {
                    const float sy = ys[yn];
                    const float4* e = yt + yn * N;
                    const float alt = (lane & 1) ? -1.f : 1.f;     // (-1)^x
#pragma unroll 1
                    for (int r = 0; r < ntask; ++r) {
                        const int kz = kz_of(r);
                        float2 vr[N], vi[N];
                        if (r == 2) {
#pragma unroll
                            for (int k = 0; k < N; ++k) {
                                const float4 v = ab16[k * N + lane];
                                vr[k] = f2(v.x, v.y);
                                vi[k] = f2(v.z, v.w);
                            }
                        } else {
#pragma unroll
                            for (int c = 0; c < N / 8; ++c) {
                                uint32_t u[16], w[16];
                                tc::tmem_ld16_issue(tab + 128 * r + 32 * c, u);
                                tc::tmem_ld16_issue(tab + 128 * r + 32 * c + 16, w);
                                tc::tmem_wait();
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    vr[8 * c + k] = f2(__uint_as_float(u[4 * k]), __uint_as_float(u[4 * k + 1]));
                                    vi[8 * c + k] = f2(__uint_as_float(u[4 * k + 2]), __uint_as_float(u[4 * k + 3]));
                                    vr[8 * c + 4 + k] = f2(__uint_as_float(w[4 * k]), __uint_as_float(w[4 * k + 1]));
                                    vi[8 * c + 4 + k] = f2(__uint_as_float(w[4 * k + 2]), __uint_as_float(w[4 * k + 3]));
                                }
                            }
                        }
                        const float2 nr = vr[H], ni = vi[H];       // at ky = N/2, before the shift
#pragma unroll
                        for (int k = 0; k < N; ++k) rot(e[k], vr[k], vi[k]);
                        {
                            const float2 v = fh[N + kz];
                            const float w = -alt * sx * sy;
                            vr[H].x += w * v.x; vr[H].y += w * v.x;
                            vi[H].x += w * v.y; vi[H].y += w * v.y;
                        }
                        if (r == 2) {                              // the field that s_z multiplies
                            const float w = alt * sx;
                            const float2 Gp = f2(w, -w), nG = f2(-w, w);
#pragma unroll
                            for (int k = 0; k < N; ++k) {
                                const float2 v = fh[k];
                                float2 pr = f2(v.x, v.x), qi = f2(v.y, v.y);
                                rot(e[k], pr, qi);
                                vr[k] = __ffma2_rn(nG, qi, vr[k]);
                                vi[k] = __ffma2_rn(Gp, pr, vi[k]);
                            }
                            vr[H] = __ffma2_rn(f2(-sy, sy), ni, vr[H]);
                            vi[H] = __ffma2_rn(f2(sy, -sy), nr, vi[H]);
                        }
                        dft_p2<N, +1>(vr, vi);
                        if (r == 0) wait_free();
                        put_z(kz, vr, vi);
                    }
                    __syncthreads();
                    const int l0 = yn ? pl.yend[yn - 1] : 0, l1 = pl.yend[yn];
#pragma unroll 1
                    for (int l = l0; l < l1; ++l) {
                        const float wr = 0.5f * float(pl.wp[l] + pl.wm[l]), wi = 0.5f * float(pl.wp[l] - pl.wm[l]);
                        const bool pair = wr == 1.f && wi == 0.f;
                        const float4* ez = zt + l * HP;
#pragma unroll 1
                        for (int j = 0; j < 4; ++j) {
                            float2 vr[N], vi[N];
#pragma unroll
                            for (int k = 0; k <= H; ++k) {
                                const float4 v = get_z(j, k);
                                vr[k] = f2(v.x, v.y);
                                vi[k] = f2(v.z, v.w);
                            }
                            if (j == 3 && l + 1 == l1) arrive();
#pragma unroll
                            for (int k = 1; k < H; ++k) {
                                const float4 m = ez[k];
                                vr[N - k] = __fmul2_rn(vr[k], f2(m.z, m.w));
                                vi[N - k] = __fmul2_rn(vi[k], f2(-m.z, -m.w));
                                vr[k] = __fmul2_rn(vr[k], f2(m.x, m.y));
                                vi[k] = __fmul2_rn(vi[k], f2(m.x, m.y));
                            }
                            vr[H] = __fmul2_rn(vr[H], f2(ez[H].x, ez[H].y));
                            vi[H] = __fmul2_rn(vi[H], f2(ez[H].z, ez[H].w));
                            float4* S = Sp + (warp + 8 * j) * N;   // + (z / 4) * N * N
                            dft_p2<N, +1>(vr, vi);
#pragma unroll
                            for (int z = 0; z < N; z += 4) {
                                float4 s = make_float4(0.f, 0.f, 0.f, 0.f);
                                if (!first) s = S[(z / 4) * N * N];
                                float t[4] = {s.x, s.y, s.z, s.w};
#pragma unroll
                                for (int k = 0; k < 4; ++k) {
                                    const float re = fmaf(vr[z + k].x, vr[z + k].y, -vi[z + k].x * vi[z + k].y);
                                    if (pair) {
                                        t[k] += re;
                                    } else {
                                        const float im = vr[z + k].x * vi[z + k].y - vi[z + k].x * vr[z + k].y;
                                        t[k] = fmaf(wr, re, fmaf(wi, im, t[k]));
                                    }
                                }
                                S[(z / 4) * N * N] = make_float4(t[0], t[1], t[2], t[3]);
                            }
                        }
                        first = false;
                    }
                }
            }

            // ---- G^ += gw_p FFT(S_p); S is half the sum, the transform doubles it ----
            forward_zy([&](int j, float (&u)[N]) {
                const float4* S = Sp + (warp + 8 * j) * N;
#pragma unroll
                for (int z = 0; z < N; z += 4) {
                    const float4 s = S[(z / 4) * N * N];
                    u[z] = s.x; u[z + 1] = s.y; u[z + 2] = s.z; u[z + 3] = s.w;
                }
            });
            const bool acc = ns == 1 && p > 0;
            auto gain = [&](float2* to, float w, float re, float im) {
                const float2 o = acc ? *to : f2(0.f, 0.f);
                *to = f2(__fadd_rn(o.x, __fmul_rn(w, re)), __fadd_rn(o.y, __fmul_rn(w, im)));
            };
            {
                float2 vr[N], vi[N];
                forward_pair(vr, vi);
                if (warp > 0) arrive();
#pragma unroll
                for (int h = 0; h < 2; ++h) {
                    const int kz = warp + 8 * h;
                    const float* gwp = gw + (size_t(p) * N + kz) * HP * N + lane;
#pragma unroll
                    for (int k = 0; k < N; ++k)
                        gain(G + k * ROW + kz * N, ldg(gwp + (k <= H ? k : N - k) * N), h ? vr[k].y : vr[k].x, h ? vi[k].y : vi[k].x);
                }
            }
            if (warp == 0) {
                cpx<float> X[N];
                forward_16(X);
                arrive();
                const float* gwp = gw + (size_t(p) * N + H) * HP * N + lane;
#pragma unroll
                for (int k = 0; k < N; ++k) gain(G + k * ROW + H * N, ldg(gwp + (k <= H ? k : N - k) * N), X[k].x, X[k].y);
            }
            if (ns > 1) G += N * ROW;
        }

        const float2* G0 = G;                                      // of the first radius, or the sum
        if (ns > 1) {
            // the part that arrives last adds the radii in order and finishes the
            // distribution
            if (s_lost) G[warp * N - N * ROW].x = tc::lost_nan(&s_lost, 0.f);
            __threadfence();
            __syncthreads();
            if (tid == 0) s_last = atomicAdd(a.tickets + it.cut, 1u) == uint32_t(ns - 1);
            __syncthreads();
            if (!s_last) continue;
            __threadfence();
            G0 = reinterpret_cast<const float2*>(a.slots + size_t(a.split.nctas + it.cut * Nrho) * QLayoutTree32::slot_bytes()) + lane;
        }

        // ---- lane A: QG = IFFT(G^), lane B: fC = IFFT(bb2 F) ----
        wait_free();
#pragma unroll 1
        for (int r = 0; r < ntask; ++r) {
            const int kz = kz_of(r);
            float2 vr[N], vi[N];
#pragma unroll
            for (int k = 0; k < N; ++k) vr[k].x = vi[k].x = 0.f;
#pragma unroll 1
            for (int j = 0; j < (ns > 1 ? Nrho : 1); ++j) {
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const float2 v = __ldcg(G0 + size_t(j) * N * ROW + k * ROW + kz * N);
                    vr[k].x = __fadd_rn(vr[k].x, v.x);
                    vi[k].x = __fadd_rn(vi[k].x, v.y);
                }
            }
#pragma unroll
            for (int k = 0; k < N; ++k) {
                const float2 v = F[k * ROW + kz * N];
                const float w = ldg(bb2 + (kz * N + k) * N + lane);
                vr[k].y = w * v.x;
                vi[k].y = w * v.y;
            }
            dft_p2<N, +1>(vr, vi);
            turn(vr, vi);
            if (r + 1 == ntask) arrive();
            dft_p2<N, +1>(vr, vi);
            // tensor memory is free: hold the y-pass results until every warp has turned
            if (r == 2) {
#pragma unroll
                for (int k = 0; k < N; ++k) ab16[k * N + lane] = make_float4(vr[k].x, vr[k].y, vi[k].x, vi[k].y);
            } else {
#pragma unroll
                for (int c = 0; c < N / 4; ++c) {
                    uint32_t u[16];
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        u[4 * k] = __float_as_uint(vr[4 * c + k].x);
                        u[4 * k + 1] = __float_as_uint(vr[4 * c + k].y);
                        u[4 * k + 2] = __float_as_uint(vi[4 * c + k].x);
                        u[4 * k + 3] = __float_as_uint(vi[4 * c + k].y);
                    }
                    tc::tmem_st16(tab + 128 * r + 16 * c, u);
                }
            }
        }
        tc::tmem_wait_st();
        wait_free();
#pragma unroll 1
        for (int r = 0; r < ntask; ++r) {
            float2 vr[N], vi[N];
            if (r == 2) {
#pragma unroll
                for (int k = 0; k < N; ++k) {
                    const float4 v = ab16[k * N + lane];
                    vr[k] = f2(v.x, v.y);
                    vi[k] = f2(v.z, v.w);
                }
            } else {
#pragma unroll
                for (int c = 0; c < N / 4; ++c) {
                    uint32_t u[16];
                    tc::tmem_ld16_issue(tab + 128 * r + 16 * c, u);
                    tc::tmem_wait();
#pragma unroll
                    for (int k = 0; k < 4; ++k) {
                        vr[4 * c + k] = f2(__uint_as_float(u[4 * k]), __uint_as_float(u[4 * k + 1]));
                        vi[4 * c + k] = f2(__uint_as_float(u[4 * k + 2]), __uint_as_float(u[4 * k + 3]));
                    }
                }
            }
            put_z(kz_of(r), vr, vi);
        }
        __syncthreads();
        const float prefac = float(g.prefac);
        double* mom = bt.moments ? bt.moments + dof * 10 : nullptr;
        const bool need_m = project || mom;
        float* Q = static_cast<float*>(bt.Q) + dof * n;
        const bool qvec = (reinterpret_cast<uintptr_t>(Q) & 15u) == 0;
        double m[5] = {0, 0, 0, 0, 0};
        const double cx = g.c0[lane];
        auto store_row = [&](float* q, const float (&u)[N]) {
            if (qvec) {
#pragma unroll
                for (int z = 0; z < N; z += 4)
                    *reinterpret_cast<float4*>(q + z) = make_float4(u[z], u[z + 1], u[z + 2], u[z + 3]);
            } else {
#pragma unroll
                for (int z = 0; z < N; ++z) q[z] = u[z];
            }
        };
#pragma unroll 1
        for (int j = 0; j < 4; ++j) {
            float2 vr[N], vi[N];
#pragma unroll
            for (int k = 0; k <= H; ++k) {
                const float4 v = get_z(j, k);
                vr[k] = f2(v.x, v.y);
                vi[k] = f2(v.z, v.w);
                if (k > 0 && k < H) {
                    vr[N - k] = vr[k];
                    vi[N - k] = f2(-v.z, -v.w);
                }
            }
            if (j == 3) arrive();
            vr[0].x = tc::lost_nan(&s_lost, vr[0].x);
            dft_p2<N, +1>(vr, vi);
            float u[N];
            load_row(f + row_at(j), fvec, u);
            double q0 = 0.0, q1 = 0.0, q2 = 0.0;
#pragma unroll
            for (int z = 0; z < N; ++z) {
                u[z] = prefac * (vr[z].x - u[z] * vr[z].y);
                if (need_m) {
                    const double cz = g.c0[z], d = double(u[z]);
                    q0 += d;
                    q1 += cz * d;
                    q2 += cz * cz * d;
                }
            }
            const double cy = g.c0[warp + 8 * j];
            m[0] += q0;
            m[1] += cx * q0;
            m[2] += cy * q0;
            m[3] += q1;
            m[4] += (cx * cx + cy * cy) * q0 + q2;
            store_row(Q + row_at(j), u);
        }
        if (need_m) block_sum<5>(m, red);
        double m2[5] = {0, 0, 0, 0, 0};
        if (project) {
            double lam[5];
#pragma unroll
            for (int i = 0; i < 5; ++i) {
                double s = 0.0;
#pragma unroll
                for (int k = 0; k < 5; ++k) s += g.ginv[i * 5 + k] * m[k];
                lam[i] = s;
            }
#pragma unroll 1
            for (int j = 0; j < 4; ++j) {                          // the thread's own rows
                const double cy = g.c0[warp + 8 * j];
                const double base = lam[0] + lam[1] * cx + lam[2] * cy + lam[4] * (cx * cx + cy * cy);
                float u[N];
                load_row(Q + row_at(j), qvec, u);
                double q0 = 0.0, q1 = 0.0, q2 = 0.0;
#pragma unroll
                for (int z = 0; z < N; ++z) {
                    const double cz = g.c0[z];
                    const double qc = double(u[z]) - (base + (lam[3] + lam[4] * cz) * cz);
                    u[z] = float(qc);
                    q0 += qc;
                    q1 += cz * qc;
                    q2 += cz * cz * qc;
                }
                m2[0] += q0;
                m2[1] += cx * q0;
                m2[2] += cy * q0;
                m2[3] += q1;
                m2[4] += (cx * cx + cy * cy) * q0 + q2;
                store_row(Q + row_at(j), u);
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
        tc::tmem_dealloc(s_tmem, 512);
    }
}

}  // namespace bdgfs
