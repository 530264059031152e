// anygrid.cuh -- the split-line passes for grids without compiled kernels of
// their own: uneven ones, and cubic sizes outside TCG_FAST_SIZES.
//
// Same algorithm and layouts as split.cuh, with the lengths n_d = a_d b_d
// (2 <= a_d, b_d <= 9) as run-time values: a short DFT is chosen by a switch that
// is uniform over the grid, its operands stay in registers (9 of them, unused
// ones predicated off).  The generic passes (passes.cuh) run one shared-memory
// sweep and one barrier per radix and remain for lengths that do not factor so.
// A TC state and apply on 20 x 18 x 21 with two spins in FP64: 19.3 ms with them,
// 12.7 with these.
// MT: most threads of an XY CTA (256: up to 255 registers, FP64 without spills;
// sl::MAXTHR for longer lines).
#pragma once
#include "terms.cuh"
#include "split.cuh"

namespace tcg {
namespace anyg {

constexpr int MX = 9;                // longest short DFT

template <typename V, int DIR> __device__ __forceinline__ void dft(int n, V (&v)[MX])
{
    switch (n) {
    case 2: sl::dft<V, 2, DIR>(v); break;
    case 3: sl::dft<V, 3, DIR>(v); break;
    case 4: sl::dft<V, 4, DIR>(v); break;
    case 5: sl::dft<V, 5, DIR>(v); break;
    case 6: sl::dft<V, 6, DIR>(v); break;
    case 7: sl::dft<V, 7, DIR>(v); break;
    case 8: sl::dft<V, 8, DIR>(v); break;
    default: sl::dft<V, 9, DIR>(v); break;
    }
}

// step 1 of thread t of a line of p * q points: DFT_q, twiddles (tw: shared), exchange
template <typename V, int DIR>
__device__ __forceinline__ void first(V *buf, int stride, int t, int p, int q, V (&u)[MX], const V *tw)
{
    dft<V, DIR>(q, u);
#pragma unroll
    for (int k = 0; k < MX; k++)
        if (k < q) {
            const V w = tw[t * k];
            buf[(k * p + t) * stride] = DIR < 0 ? cmul(u[k], w) : cmulc(w, u[k]);
        }
}
template <typename V, int DIR> __device__ __forceinline__ void second(const V *buf, int stride, int t, int p, V (&v)[MX])
{
#pragma unroll
    for (int j = 0; j < MX; j++)
        if (j < p) v[j] = buf[(t * p + j) * stride];
    dft<V, DIR>(p, v);
}

// Threads of an XY CTA: phase y works on lines along y (lane x), phase x on lines along x (lane y)
struct XY {
    int n0, n1, a0, b0, a1, b1, ty, lx, tx, ly;   // ty, lx: thread / lane of phase y; tx, ly of phase x
    int rs;                                        // row stride of a buffer (odd)
    __device__ __forceinline__ void init(const sl::AnyShape &s)
    {
        n0 = s.n[0]; n1 = s.n[1];
        a0 = s.a[0]; b0 = s.b[0]; a1 = s.a[1]; b1 = s.b[1];
        ty = threadIdx.x / n0; lx = threadIdx.x % n0;
        tx = threadIdx.x / n1; ly = threadIdx.x % n1;
        rs = s.rs;
    }
};

// forward: u[m] = f(x = lx, y = ty + a1 m), ty < a1 -> v[m] = F(kx = tx + b0 m, ky = ly), tx < b0
template <typename V>
__device__ __forceinline__ void plane_fwd(const XY &g, V *b0, V *b1, V (&u)[MX], const V *twx, const V *twy, V (&v)[MX])
{
    if (g.ty < g.a1) first<V, -1>(b0 + g.lx, g.rs, g.ty, g.a1, g.b1, u, twy);
    __syncthreads();
    if (g.ty < g.b1) {
        second<V, -1>(b0 + g.lx, g.rs, g.ty, g.a1, v);
#pragma unroll
        for (int m = 0; m < MX; m++)
            if (m < g.a1) b1[(g.ty + g.b1 * m) * g.rs + g.lx] = v[m];
    }
    __syncthreads();
    if (g.tx < g.a0) {
#pragma unroll
        for (int m = 0; m < MX; m++)
            if (m < g.b0) u[m] = b1[g.ly * g.rs + g.tx + g.a0 * m];
        first<V, -1>(b0 + g.ly, g.rs, g.tx, g.a0, g.b0, u, twx);
    }
    __syncthreads();
    if (g.tx < g.b0) second<V, -1>(b0 + g.ly, g.rs, g.tx, g.a0, v);
}
// inverse: u[m] = F(kx = tx + b0 m, ky = ly), tx < b0 -> v[m] = f(x = lx, y = ty + a1 m), ty < a1
template <typename V>
__device__ __forceinline__ void plane_inv(const XY &g, V *b0, V *b1, V (&u)[MX], const V *twx, const V *twy, V (&v)[MX])
{
    if (g.tx < g.b0) first<V, +1>(b0 + g.ly, g.rs, g.tx, g.b0, g.a0, u, twx);
    __syncthreads();
    if (g.tx < g.a0) {
        second<V, +1>(b0 + g.ly, g.rs, g.tx, g.b0, v);
#pragma unroll
        for (int m = 0; m < MX; m++)
            if (m < g.b0) b1[g.ly * g.rs + g.tx + g.a0 * m] = v[m];
    }
    __syncthreads();
    if (g.ty < g.b1) {
#pragma unroll
        for (int m = 0; m < MX; m++)
            if (m < g.a1) u[m] = b1[(g.ty + g.b1 * m) * g.rs + g.lx];
        first<V, +1>(b0 + g.lx, g.rs, g.ty, g.b1, g.a1, u, twy);
    }
    __syncthreads();
    if (g.ty < g.a1) second<V, +1>(b0 + g.lx, g.rs, g.ty, g.b1, v);
}

template <typename V> __device__ __forceinline__ void stage_axis(const GridDesc &g, int d, V *dst)
{
    const V *src = twsrc<V>(g) + d * MAXN;
    for (int i = threadIdx.x; i < g.ax[d].n; i += blockDim.x) dst[i] = src[i];
}

template <typename T, class Op, int MT>
__global__ void __launch_bounds__(MT) k_xyf(Op op, sl::AnyShape S, int items)
{
    using V = typename C2<T>::t;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *twx = reinterpret_cast<V *>(smem_raw), *twy = twx + S.n[0];
    V *b0 = twy + S.n[1], *b1 = b0 + S.ps;
    stage_axis<V>(op.g, 0, twx);
    stage_axis<V>(op.g, 1, twy);
    XY g;
    g.init(S);
    const int z = blockIdx.x / items, item = blockIdx.x % items;
    const size_t plane = (size_t)g.n0 * g.n1, pz = z * plane;
    unsigned long long bits = ~0ull;
    if (Op::BLI != 0 && op.m.prune && g.tx < g.b0) bits = op.pcol(item, g.ly);
    __syncthreads();
#pragma unroll 1
    for (int f = 0; f < Op::NF; f++) {
        V u[MX], v[MX];
        if (g.ty < g.a1) {
#pragma unroll
            for (int m = 0; m < MX; m++)
                if (m < g.b1) {
                    const int y = g.ty + g.a1 * m;
                    u[m] = op.xyf_load(item, f, g.lx, y, z, pz + (size_t)y * g.n0 + g.lx);
                }
        }
        plane_fwd<V>(g, b0, b1, u, twx, twy, v);
        if (g.tx < g.b0) {
            V *dst = op.tmp_grid(item, f) + pz + g.ly;
            const bool bl = (Op::BLI >> f) & 1;
#pragma unroll
            for (int m = 0; m < MX; m++)
                if (m < g.a0 && (!bl || ((bits >> (g.tx + g.b0 * m)) & 1))) dst[(size_t)(g.tx + g.b0 * m) * g.n1] = v[m];
        }
        V *s = b0;
        b0 = b1;
        b1 = s;
    }
}

template <typename T, class Op, int MT>
__global__ void __launch_bounds__(MT) k_xyi(Op op, sl::AnyShape S, int nt)
{
    using V = typename C2<T>::t;
    constexpr int NA = Op::NACC;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *twx = reinterpret_cast<V *>(smem_raw), *twy = twx + S.n[0];
    V *b0 = twy + S.n[1], *b1 = b0 + S.ps;
    V *acc = b1 + S.ps + threadIdx.x;            // [NA][b1][threads] sums of this thread's points
    stage_axis<V>(op.g, 0, twx);
    stage_axis<V>(op.g, 1, twy);
    XY g;
    g.init(S);
    const int z = blockIdx.x / nt, tj = blockIdx.x % nt;
    const size_t plane = (size_t)g.n0 * g.n1, pz = z * plane, p0 = pz + (size_t)g.ty * g.n0 + g.lx;
    const int ns = op.nsrc(tj), nthr = blockDim.x;
    const size_t ystep = (size_t)g.a1 * g.n0, xstep = (size_t)g.b0 * g.n1;
    const bool mine = g.ty < g.a1;
    for (int a = 0; a < NA * g.b1; a++) acc[a * nthr] = czero<V>();
    __syncthreads();
    V keep[Op::GS][MX];
    // G plane b of source si: where the CTA is small (registers to spare) the next one
    // is on its way while the current one is transformed (the spin-polarised TC state
    // and apply on 20 x 18 x 21 14.2 -> 12.7 ms)
    constexpr bool AHEAD = MT <= 256;
    V nx[AHEAD ? MX : 1];
    auto fetch = [&](int si, int b, V *u) {
        if (g.tx >= g.b0) return;
        const int item = op.item_of(tj, si);
        const V *src = op.xyi_grid(item, b) + pz + (size_t)g.tx * g.n1 + g.ly;
        const bool bl = op.m.prune && ((Op::BLO >> b) & 1);
        const unsigned long long bits = bl ? op.pcol(item, g.ly) >> g.tx : ~0ull;
#pragma unroll
        for (int m = 0; m < MX; m++)
            if (m < g.a0) u[m] = (bits >> (g.b0 * m)) & 1 ? src[m * xstep] : czero<V>();
    };
    if constexpr (AHEAD) fetch(0, 0, nx);
#pragma unroll 1
    for (int bg = 0; bg < Op::NB; bg += Op::GS) {
#pragma unroll 1
        for (int si = 0; si < ns; si++) {
            const int item = op.item_of(tj, si);
            unsigned long long bits = ~0ull;
            if (op.m.prune && g.tx < g.b0) bits = op.pcol(item, g.ly);
            V v[MX];
#pragma unroll
            for (int q = 0; q < Op::GS; q++) {
                V u[MX];
                if constexpr (AHEAD) {
#pragma unroll
                    for (int m = 0; m < MX; m++) u[m] = nx[m];
                    if (q + 1 < Op::GS) fetch(si, bg + q + 1, nx);
                    else if (si + 1 < ns) fetch(si + 1, bg, nx);
                    else if (bg + Op::GS < Op::NB) fetch(0, bg + Op::GS, nx);
                } else if (g.tx < g.b0) {
                    const V *src = op.xyi_grid(item, bg + q) + pz + (size_t)g.tx * g.n1 + g.ly;
                    const bool bl = (Op::BLO >> (bg + q)) & 1;
#pragma unroll
                    for (int m = 0; m < MX; m++)
                        if (m < g.a0)
                            u[m] = !bl || ((bits >> (g.tx + g.b0 * m)) & 1) ? src[m * xstep] : czero<V>();
                }
                plane_inv<V>(g, b0, b1, u, twx, twy, v);
                V *s = b0;
                b0 = b1;
                b1 = s;
                if (q < Op::GS - 1) {
#pragma unroll
                    for (int m = 0; m < MX; m++) keep[q][m] = v[m];
                }
            }
            if (mine) {
#pragma unroll
                for (int m = 0; m < MX; m++)
                    if (m < g.b1) {
                        V vals[Op::GS], o[Op::NOPS];
#pragma unroll
                        for (int q = 0; q < Op::GS - 1; q++) vals[q] = keep[q][m];
                        vals[Op::GS - 1] = v[m];
#pragma unroll
                        for (int k = 0; k < Op::NOPS; k++) {
                            const V *src = op.xyi_operand(k, bg, si);
                            o[k] = src ? __ldg(src + p0 + m * ystep) : czero<V>();
                        }
                        op.xyi_add(si, bg, vals, o, [&](int slot, V x) {
                            V *a = acc + (slot * g.b1 + m) * nthr;
                            *a = cadd(*a, x);
                        });
                    }
            }
            if (mine && (si + 1 == ns || sl::flush_due<V>(si)))
                for (int a = 0; a < NA; a++)
#pragma unroll
                    for (int m = 0; m < MX; m++)
                        if (m < g.b1) {
                            V *s = acc + (a * g.b1 + m) * nthr;
                            op.xyi_put(tj, bg, a, p0 + m * ystep, *s);
                            *s = czero<V>();
                        }
            if (Op::REFWD && op.refwd_want(bg)) {
                if (mine) {
#pragma unroll
                    for (int m = 0; m < MX; m++)
                        if (m < g.b1) v[m] = op.refwd_load(tj, item, bg, p0 + m * ystep, v[m]);
                }
                V w[MX];
                plane_fwd<V>(g, b0, b1, v, twx, twy, w);
                V *s = b0;
                b0 = b1;
                b1 = s;
                if (g.tx < g.b0) {
                    V *dst = op.refwd_grid(item, bg) + pz + (size_t)g.tx * g.n1 + g.ly;
#pragma unroll
                    for (int m = 0; m < MX; m++)
                        if (m < g.a0 && (!op.m.prune || ((bits >> (g.tx + g.b0 * m)) & 1))) dst[m * xstep] = w[m];
                }
            }
        }
    }
}

// one item, TC consecutive pencils, a threads per z-line
template <typename T, class Op> __global__ void __launch_bounds__(9 * 32) k_z(Op op, sl::AnyShape S)
{
    using V = typename C2<T>::t;
    constexpr int TC = 32, NF = Op::NF, ZK = Op::ZK;
    const int n = S.n[2], A = S.a[2], B = S.b[2], np = S.n[0] * S.n[1];
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw), *E = tw + n;     // [max(NF, 2)][n][TC]
    stage_axis<V>(op.g, 2, tw);
    const int item = blockIdx.y, t = threadIdx.x / TC, cl = threadIdx.x % TC, slot = blockIdx.x * TC + cl;
    const bool prune = op.m.prune != 0;
    int c = slot;
    bool allin = false, pon = true;
    if (prune) {
        const int e = op.pent_of(item), na = op.m.pnact[e];
        if (slot < np) c = op.m.pperm[(size_t)e * op.m.np + slot];
        allin = blockIdx.x * TC >= na;
        pon = slot < na;
        constexpr unsigned FI = (1u << NF) - 1, FO = (1u << Op::NB) - 1;
        if (allin && (Op::BLI & FI) == FI && (Op::BLO & FO) == FO) return;
    }
    const bool act = slot < np;
    const auto zc = op.zctx(item, c / S.n[1], c % S.n[1], c);   // y fastest (m.tr)
    __syncthreads();
#pragma unroll 1
    for (int f = 0; f < NF; f++) {
        V u[MX];
        const bool rd = act && (!(prune && ((Op::BLI >> f) & 1)) || pon);
        const V *src = op.zin_grid(item, f) + c;
#pragma unroll
        for (int m = 0; m < MX; m++)
            if (m < B) u[m] = rd ? src[(size_t)(t + A * m) * np] : czero<V>();
        first<V, -1>(E + f * n * TC + cl, TC, t, A, B, u, tw);
    }
    __syncthreads();
    V K[ZK][MX], mix[MX];
    if (t < B) {
#pragma unroll
        for (int f = 0; f < NF; f++) {
            V X[MX];
            second<V, -1>(E + f * n * TC + cl, TC, t, A, X);
#pragma unroll
            for (int m = 0; m < MX; m++)
                if (m < A) {
                    if (f < ZK) K[f < ZK ? f : 0][m] = X[m];
                    if (Op::ZMO >= 0 && f >= Op::ZM0) {
                        const V w = cscale(X[m], act ? op.zmixc(zc, f, t + B * m) : (T)0);
                        mix[m] = f == Op::ZM0 ? w : cadd(mix[m], w);
                    }
                }
        }
    }
    __syncthreads();
    int buf = 0;
#pragma unroll 1
    for (int i = 0; i < Op::NB; i++) {
        const int o = Op::ZMO > 0 ? (i == 0 ? Op::ZMO : (i <= Op::ZMO ? i - 1 : i)) : i;
        const bool blo = prune && ((Op::BLO >> o) & 1);
        if (blo && allin) continue;
        V v[MX];
        if (t < B) {
            const int k = op.zsrc(o);
#pragma unroll
            for (int m = 0; m < MX; m++)
                if (m < A) {
                    if (o == Op::ZMO) v[m] = mix[m];
                    else v[m] = cscale(ZK > 1 && k ? K[ZK - 1][m] : K[0][m], act ? op.zoutc(zc, o, t + B * m) : (T)0);
                }
        }
        V *dst = op.out_grid(item, o) + c;
        if (Op::ZINV) {
            V *Eo = E + buf * n * TC + cl;
            buf ^= 1;
            if (t < B) first<V, +1>(Eo, TC, t, B, A, v, tw);
            __syncthreads();
            V r[MX];
            second<V, +1>(Eo, TC, t, B, r);
            if (act && (!blo || pon)) {
#pragma unroll
                for (int m = 0; m < MX; m++)
                    if (m < B) dst[(size_t)(t + A * m) * np] = r[m];
            }
        } else if (act && t < B && (!blo || pon)) {
#pragma unroll
            for (int m = 0; m < MX; m++)
                if (m < A) dst[(size_t)(t + B * m) * np] = v[m];
        }
    }
}

} // namespace anyg
} // namespace tcg
