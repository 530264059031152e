// terms.cuh -- operator terms on top of the pass kernels.
//
//   hf2x         calc_hamiltonian_hf2x.cpp:8-205
//   tc2x         calc_hamiltonian_tc2x.cpp:11-516   (SCF mesh: kVaux = 0)
//   tc3a1, tc3b1 calc_hamiltonian_tc3a1.cpp:8-117, tc3b1.cpp:8-135
//   tc3a3b3b4b6  calc_hamiltonian_tc3a3b3b4b6.cpp:11-863
//   tc3a2a4b2b5  calc_hamiltonian_tc3a2a4b2b5.cpp:11-1300
//
// Every exchange-like sum  sum_{q,i} f_qi X_qi(r) IFFT[K(k-q+G) FFT[Y_qi(r) Z_kj(r)]]
// runs as chunks of (target bands) x (occupied sources) through the three
// fused passes (passes.cuh).  All R-space contributions to H2 psi (resp.
// H3 psi) of one band are summed in one FP64 accumulator and transformed /
// gathered onto the sphere once at the end.  Work that depends only on the
// occupied orbitals (R-space orbitals and gradients, the local three-body
// potentials of tc3a1 / tc3b1 / tc3a2 / tc3b2, and the occupied-pair stage of
// tc3a2a4b2b5 with its symmetry-rotated intermediates) is done once per
// tcg_set_state: TC++ recomputes it inside every calc_hamiltonian::all call,
// although BlochStates is constant across the calls of one Davidson step.
#pragma once
#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>
#include "ctx.cuh"
#include "passes.cuh"
#include "util.cuh"
#include "jastrow.cuh"

namespace tcg {

struct ApplyArgs {
    uint32_t mask;
    const int32_t *nb;
    const uint8_t *owned;
    const double2 *psi;
    double2 *h2, *h3;
};

constexpr double PI_D = 3.14159265358979323846;

struct RecipC {
    double R[9];
};

static inline void cart(const Host &h, const double *x, double *v)
{
    for (int d = 0; d < 3; d++) v[d] = h.recip[0 * 3 + d] * x[0] + h.recip[1 * 3 + d] * x[1] + h.recip[2 * 3 + d] * x[2];
}

__device__ __forceinline__ void gvec(const double *R, const GridDesc &g, int x, int y, int z, const double *q, double *G)
{
    const int m0 = miller(x, g.n0), m1 = miller(y, g.n1), m2 = miller(z, g.n2);
#pragma unroll
    for (int d = 0; d < 3; d++) G[d] = q[d] + R[0 * 3 + d] * m0 + R[1 * 3 + d] * m1 + R[2 * 3 + d] * m2;
}

__device__ __forceinline__ void xyz_of(const GridDesc &g, size_t p, int &x, int &y, int &z)
{
    x = (int)(p % g.n0);
    y = (int)((p / g.n0) % g.n1);
    z = (int)(p / ((size_t)g.n0 * g.n1));
}

__device__ __forceinline__ void acc_add(double2 *a, double2 v, double f) { *a = {a->x + f * v.x, a->y + f * v.y}; }
// fire-and-forget accumulation (red.global.add.f64): no load / store
// round trip per update.  Every accumulator element is updated by one thread
// only, so the updates of an element keep their program order and the sum
// is deterministic.
__device__ __forceinline__ void acc_red(double2 *a, double2 v, double f)
{
    atomicAdd(&a->x, f * v.x);
    atomicAdd(&a->y, f * v.y);
}

// ------------------------------------------------- transforms of whole grids --
// The four passes of a list of transforms: on the compiled cubic sizes in split
// lines (fft_split.cuh, instantiated with the pair passes), else generic.
template <typename T, int N> struct FastIO {
    static int xy(tcg_ctx *c, const GridDesc &g, const GridRefs &gr, unsigned n, int dir);
    static int z(tcg_ctx *c, const GridDesc &g, const GridRefs &gr, unsigned n, int dir, double scale);
    static int sphere(tcg_ctx *c, const GridDesc &g, const SphereItem *items, unsigned n);
    static int gather(tcg_ctx *c, const GridDesc &g, const GatherItem *items, unsigned n);
};
static bool io_fast(const tcg_ctx *c, const GridDesc &g)
{
    return !c->force_generic && g.n0 == g.n1 && g.n1 == g.n2 && fast_grid(g.n0);
}
#define TCG_IO(T, call)                                                    \
    if (io_fast(c, g)) {                                                   \
        switch (g.n0) {                                                    \
        TCG_FAST_SIZES(TCG_IO_CASE)                                        \
        default: break;                                                    \
        }                                                                  \
    }
template <typename T, int DIR> static int grids_xy(tcg_ctx *c, const GridDesc &g, const GridRefs &gr, unsigned n)
{
#define TCG_IO_CASE(m) case m: return FastIO<T, m>::xy(c, g, gr, n, DIR);
    TCG_IO(T, xy)
#undef TCG_IO_CASE
    return launch(c, k_xy_inplace<T, DIR>, dim3(g.n2, n), dim3(256), smem_xy<typename C2<T>::t>(g), g, gr);
}
template <typename T, int DIR> static int grids_z(tcg_ctx *c, const GridDesc &g, const GridRefs &gr, unsigned n, double scale)
{
#define TCG_IO_CASE(m) case m: return FastIO<T, m>::z(c, g, gr, n, DIR, scale);
    TCG_IO(T, z)
#undef TCG_IO_CASE
    return launch(c, k_z_inplace<T, DIR>, dim3((g.n0 * g.n1 + ZTC - 1) / ZTC, n), dim3(256), smem_z<typename C2<T>::t>(g, 0), g, gr,
                  scale);
}
template <typename T> static int sphere_z(tcg_ctx *c, const GridDesc &g, const SphereItem *items, unsigned n)
{
#define TCG_IO_CASE(m) case m: return FastIO<T, m>::sphere(c, g, items, n);
    TCG_IO(T, sphere)
#undef TCG_IO_CASE
    return launch(c, k_sphere_z<T>, dim3((g.n0 * g.n1 + ZTC - 1) / ZTC, n), dim3(256), smem_z<typename C2<T>::t>(g, 0), g, items,
                  c->recip.as<const double>());
}
static int gather_z(tcg_ctx *c, const GridDesc &g, const GatherItem *items, unsigned n)
{
#define TCG_IO_CASE(m) case m: return FastIO<double, m>::gather(c, g, items, n);
    TCG_IO(double, gather)
#undef TCG_IO_CASE
    return launch(c, k_gather_z, dim3((g.n0 * g.n1 + ZTC - 1) / ZTC, n), dim3(256), smem_z<double2>(g, 0), g, items);
}

// ---------------------------------------------------------------- sphere --
template <typename T>
static int sphere_to_r(tcg_ctx *c, const std::vector<SphereItem> &items)
{
    const GridDesc &g = c->gd;
    if (items.empty()) return TCG_OK;
    const size_t n = items.size();
    std::vector<void *> outs(n);
    for (size_t i = 0; i < n; i++) outs[i] = items[i].out;
    TRY(c->items.ensure(n * (sizeof(SphereItem) + sizeof(void *))));
    SphereItem *d_items = c->items.as<SphereItem>();
    void **d_outs = reinterpret_cast<void **>(d_items + n);
    TCG_CUDA(cudaMemcpyAsync(d_items, items.data(), n * sizeof(SphereItem), cudaMemcpyHostToDevice, c->stream));
    TCG_CUDA(cudaMemcpyAsync(d_outs, outs.data(), n * sizeof(void *), cudaMemcpyHostToDevice, c->stream));
    for (size_t b0 = 0; b0 < n; b0 += 65535) {
        const unsigned nb = (unsigned)std::min<size_t>(65535, n - b0);
        TRY(sphere_z<T>(c, g, d_items + b0, nb));
        GridRefs gr;
        gr.dev = d_outs + b0;
        TRY((grids_xy<T, +1>(c, g, gr, nb)));
    }
    return TCG_OK;
}

// In-place full 3D FFT of a list of grids (DIR -1: forward with 1/N).
template <typename T, int DIR>
static int fft3_list(tcg_ctx *c, const std::vector<void *> &grids, const GridDesc *on = nullptr)
{
    const GridDesc &g = on ? *on : c->gd;
    if (grids.empty()) return TCG_OK;
    const size_t n = grids.size();
    const double scale = DIR < 0 ? 1.0 / (double)g.N : 1.0;
    if (n <= 8) {   // pointers by value: nothing to upload, nothing to wait for
        GridRefs gr;
        for (size_t i = 0; i < n; i++) gr.inl[i] = grids[i];
        TRY((grids_xy<T, DIR>(c, g, gr, (unsigned)n)));
        return grids_z<T, DIR>(c, g, gr, (unsigned)n, scale);
    }
    TRY(c->items.ensure(n * sizeof(void *)));
    void **d = c->items.as<void *>();
    TCG_CUDA(cudaMemcpyAsync(d, grids.data(), n * sizeof(void *), cudaMemcpyHostToDevice, c->stream));
    for (size_t b0 = 0; b0 < n; b0 += 65535) {
        const unsigned nb = (unsigned)std::min<size_t>(65535, n - b0);
        GridRefs gr;
        gr.dev = d + b0;
        TRY((grids_xy<T, DIR>(c, g, gr, nb)));
        TRY((grids_z<T, DIR>(c, g, gr, nb, scale)));
    }
    return TCG_OK;
}

// The same for n evenly spaced grids of N points.
template <typename T, int DIR>
static int fft3_strided(tcg_ctx *c, typename C2<T>::t *first, size_t n)
{
    using V = typename C2<T>::t;
    const GridDesc &g = c->gd;
    const double scale = DIR < 0 ? 1.0 / (double)g.N : 1.0;
    for (size_t b0 = 0; b0 < n; b0 += 65535) {
        const unsigned nb = (unsigned)std::min<size_t>(65535, n - b0);
        GridRefs gr;
        gr.base = reinterpret_cast<char *>(first + b0 * g.N);
        gr.stride = (size_t)g.N * sizeof(V);
        TRY((grids_xy<T, DIR>(c, g, gr, nb)));
        TRY((grids_z<T, DIR>(c, g, gr, nb, scale)));
    }
    return TCG_OK;
}

// --------------------------------------------------------------- targets --
struct Targets {
    std::vector<int> s, k, j;
    std::vector<size_t> psi_off;            // complex offset of the band in psi
    std::vector<int> blk;                   // block starts (equal (s,k)) + end
};

static Targets make_targets(const tcg_ctx *c, const ApplyArgs &A)
{
    const Host &h = c->h;
    Targets T;
    size_t off = 0, flat = 0;
    for (int s = 0; s < h.nspin; s++)
        for (int k = 0; k < h.nk; k++) {
            bool opened = false;
            for (int j = 0; j < A.nb[s * h.nk + k]; j++, flat++, off += h.npw[k]) {
                if (A.owned && !A.owned[flat]) continue;
                if (!opened) { T.blk.push_back((int)T.s.size()); opened = true; }
                T.s.push_back(s);
                T.k.push_back(k);
                T.j.push_back(j);
                T.psi_off.push_back(off);
            }
        }
    T.blk.push_back((int)T.s.size());
    return T;
}

// ============================================================ op plumbing ==
// Common chunk description shared by the ops: targets tj in [0, nt),
// sources si in [0, ns), item = tj * ns + si.  Each target belongs to a
// target block tb (equal k) and each source to a source block sb (equal
// all-k index); per (tb, sb) a kq vector and a Jastrow table row exist.
struct ChunkMeta {
    const int *tb;          // [nt]
    const int *sb;          // [ns]
    const double *kq;       // [nTB*nSB][3]
    const double *tab;      // [nTB*nSB][N][ntab]            (FP64 path)
    const float *ftab;      // [nTB*nSB][nrec][N] coefficients (mixed path), one plane per component
    int nSB, ntab, nrec;
    // G-side planes y fastest (split-line XY passes, split.cuh): grids between
    // the XY and Z passes and the coefficient tables
    int tr;
    // pruning (prune != 0): per pair its entry in the context's pencil table of
    // the pencils (x, y) that the ball |G + k - q| < R_k + R_q meets; pperm lists
    // the active pencils y + n1 x first, pnact counts them
    const int *pent;        // [nTB*nSB]
    const unsigned short *pperm;
    const int *pnact;
    const unsigned long long *pbits;   // [entry][y]: bit x set where pencil (x, y) is active
    int np, prune;
    double pfrac;           // mean active-pencil fraction of the chunk's items (host accounting)
    int pmax;               // most active pencils of its pairs (host: Z-pass grid)
};

template <typename T>
struct OpBase {
    using V = typename C2<T>::t;
    static constexpr bool ZINV = true, REFWD = false;
    static constexpr int GS = 1;
    static constexpr int ZMINB = 3;          // min resident CTAs of the fast Z pass (register cap)
    static constexpr bool ZSPLIT = true;     // fast Z pass: z-lines split over lane pairs
    // fast XY passes: one thread per line (measured fastest for every term on
    // 36^3 once the plane copies were made division-free) or lines split over
    // lane pairs (half the registers, one shuffle per element)
    static constexpr bool XYF_PAIR = false, XYI_PAIR = false;
    GridDesc g;
    V *tmp;
    int nsl;                // tmp slots per item
    int ns;                 // sources in the chunk
    ChunkMeta m;
    RecipC rc;
    double invN;
    __device__ V *tmp_grid(int item, int f) const { return tmp + ((size_t)item * nsl + f) * g.N; }
    __device__ V *zin_grid(int item, int f) const { return tmp_grid(item, f); }
    __device__ V *out_grid(int item, int o) const { return tmp_grid(item, o); }
    __device__ V *xyi_grid(int item, int b) const { return tmp_grid(item, b); }
    __device__ void xyf_begin(int) const {}
    __device__ void z_begin(int) const {}
    __device__ void xyi_end(int, int) const {}
    __device__ int nsrc(int) const { return ns; }
    __device__ int item_of(int tj, int si) const { return tj * ns + si; }
    __device__ bool refwd_want(int) const { return false; }
    // v times the density of output b's branch (densities refwd_dens, NRW of them)
    static constexpr int NRW = 0;
    __device__ const V *refwd_dens(int) const { return nullptr; }
    __device__ V refwd_mul(int, V v, V) const { return v; }
    __device__ V refwd_load(int, int, int, size_t, V v) const { return v; }
    __device__ V *refwd_grid(int, int) const { return nullptr; }
    __device__ V xyf_load(int, int, int, int, int, size_t) const { return czero<V>(); }
    // register accumulation (fast XYI path, FP32): grids b with regacc_grid(b)
    // contribute xyi_term(...) to a per-thread column sum flushed once per
    // chunk with xyi_flush; the other grids go through xyi_accum.
    static constexpr bool REGACC = false;
    static constexpr bool BOUTER = false;    // one register accumulator per output grid (xyi_flush_b)
    // RACC_EXTRA: besides the register sum, every output also goes to
    // xyi_extra(tj, item, b, p, v) (other accumulators of the op)
    static constexpr bool RACC_EXTRA = false;
    __device__ void xyi_extra(int, int, int, size_t, const V *) const {}
    // ---- split-line passes (split.cuh)
    // Inverse XY: the sums over the sources that an output group feeds, at most
    // NACC of them, made with at most NOPS operand grids of the source
    // (xyi_operand(k, b0, si), null where unused): xyi_add(si, b0, vals[GS], o,
    // add) calls add(slot, value) for the group b0's contributions at a point,
    // xyi_put(tj, b0, slot, p, sum) adds a finished sum to its FP64 accumulator (FP32: after
    // every sl::FLUSH sources).
    static constexpr int NACC = 1, NOPS = 1;
    __device__ const V *xyi_operand(int, int, int) const { return nullptr; }
    template <class F> __device__ void xyi_add(int, int, const V *, const V *, F &&) const {}
    __device__ void xyi_put(int, int, int, size_t, V) const {}
    // Forward XY: at most NSO operand grids of the source per input (xyf_operand(k,
    // f, si), null where unused); xyf_pair(tj, f, p, o) is the input's value from
    // them and the target's operands, the same as xyf_load.  NSO = 0: xyf_load.
    static constexpr int NSO = 1;
    // Z: output ZMO = sum over f >= ZM0 of zmixc(f) X_f, the others zoutc(o) X_zsrc(o);
    // inputs f < ZK stay in registers.  The same combination as zmix.
    static constexpr int ZK = 1, ZMO = 0, ZM0 = 0;
    __device__ int zsrc(int) const { return 0; }
    // what the coefficients of one item and pencil need, looked up once: FP32 its
    // planes at the pencil, FP64 its table column and k - q + G without the z part
    struct ZC {
        const float *ft;
        const double *td;
        double q[3];
        T f;                 // filling of the item's source (ops that use it)
    };
    __device__ ZC zctx_base(int item, int x, int y, int c, int ncol) const
    {
        ZC z;
        const int pr = pair_id(item);
        z.f = (T)1;
        if constexpr (sizeof(T) == 4) z.ft = m.ftab + (size_t)pr * m.nrec * g.N + c;
        else {
            z.td = m.tab + ((size_t)pr * g.N + c) * ncol;
            const int m0 = miller(x, g.n0), m1 = miller(y, g.n1);
#pragma unroll
            for (int d = 0; d < 3; d++) z.q[d] = m.kq[3 * pr + d] + rc.R[d] * m0 + rc.R[3 + d] * m1;
        }
        return z;
    }
    // coefficient plane r at height z (FP32); table column col and
    // (k - q + G)_d u(G)/N from u in column col (FP64, ncol columns)
    __device__ T zpl(const ZC &c, int r, int z) const { return (T)__ldg(c.ft + (size_t)r * g.N + (size_t)z * g.n0 * g.n1); }
    __device__ double zcol(const ZC &c, int ncol, int col, int z) const
    {
        return __ldg(c.td + (size_t)z * g.n0 * g.n1 * ncol + col);
    }
    __device__ double zdu(const ZC &c, int ncol, int col, int d, int z) const
    {
        const double u = zcol(c, ncol, col, z) * invN, m2 = miller(z, g.n2);
        const double k = d == 0 ? c.q[0] + rc.R[6] * m2 : (d == 1 ? c.q[1] + rc.R[7] * m2 : c.q[2] + rc.R[8] * m2);
        return k * u;
    }
    __device__ bool regacc_grid(int) const { return false; }
    __device__ V xyi_term(int, int, int, size_t, const V *v) const { return v[0]; }
    __device__ void xyi_flush(int, size_t, V) const {}
    __device__ int pair_id(int item) const { return m.tb[item / ns] * m.nSB + m.sb[item % ns]; }
    __device__ const double *kq_of(int item) const { return m.kq + 3 * pair_id(item); }
    __device__ const double *tab_of(int item) const { return m.tab + (size_t)pair_id(item) * g.N * m.ntab; }
    // mixed path: plane r of the coefficient table at grid point p.  (One plane
    // per component: an output that needs one of them reads 4 bytes per point,
    // not a record of 16, from tables that stay in L2.)
    __device__ float fco(int item, size_t p, int r) const
    {
        return __ldg(&m.ftab[((size_t)pair_id(item) * m.nrec + r) * g.N + p]);
    }
    static constexpr bool FT = sizeof(T) == 4;   // mixed path: FP32 coefficient tables
    // index of G-space point (x, y, z) in the grids between the passes and the tables
    __device__ size_t pidx(int x, int y, int z) const
    {
        return m.tr ? (size_t)y + (size_t)g.n1 * (x + (size_t)g.n0 * z) : (size_t)x + (size_t)g.n0 * (y + (size_t)g.n1 * z);
    }
    // Inputs (bit f of BLI) and outputs (bit o of BLO) of which only the pencils
    // inside the ball |G + k - q| < R_k + R_q are needed; with m.prune set, the
    // pass kernels skip the others (XYF stores, Z loads / transforms / stores,
    // XYI loads read as zero).  Two kinds: pair densities conj(a_q) b_k of two
    // orbitals of the plane-wave spheres of q and k and their G-space multiples,
    // which vanish outside it; and grids X of terms phi_q(r) X(r) (or with
    // grad phi_q) that are only gathered on the sphere of k, since a component G
    // of X reaches k + G' only through q + G' - G inside the sphere of q.
    static constexpr unsigned BLI = 0, BLO = 0;
    __device__ int pent_of(int item) const { return m.pent[pair_id(item)]; }
    // active x of row y of the item's pair (bit x)
    __device__ unsigned long long pcol(int item, int y) const { return m.pbits[(size_t)pent_of(item) * g.n1 + y]; }
};

// =================================================================== hf2x ==
template <typename T>
struct OpHF2X : OpBase<T> {
    using V = typename C2<T>::t;
    static constexpr const char *NAME = "hf2x";
    static constexpr unsigned BLI = 1, BLO = 1;
    static constexpr bool REGACC = true;
    __device__ bool regacc_grid(int) const { return true; }
    __device__ V xyi_term(int, int item, int, size_t p, const V *v) const
    {
        const int si = item % this->ns;
        return cscale(cmul(v[0], __ldg(&Rocc[(size_t)si * this->g.N + p])), (decltype(v[0].x))fill[si]);
    }
    __device__ void xyi_flush(int tj, size_t p, V s) const { acc_red(acc + (size_t)tj * this->g.N + p, to64(s), 1.0); }
    __device__ const V *xyi_operand(int, int, int si) const { return Rocc + (size_t)si * this->g.N; }
    template <class F> __device__ void xyi_add(int si, int, const V *v, const V *o, F &&add) const
    {
        add(0, cscale64(cmul(v[0], o[0]), fill[si]));
    }
    __device__ const V *xyf_operand(int, int, int si) const { return Rocc + (size_t)si * this->g.N; }
    __device__ V xyf_pair(int tj, int, size_t p, const V *o) const { return cmulc(o[0], __ldg(&Rpsi[(size_t)tj * this->g.N + p])); }
    using ZC = typename OpBase<T>::ZC;
    __device__ ZC zctx(int item, int x, int y, int c) const { return this->zctx_base(item, x, y, c, 1); }
    __device__ T zmixc(const ZC &c, int, int z) const
    {
        if constexpr (OpBase<T>::FT) return this->zpl(c, 0, z);
        else return this->zcol(c, 1, 0, z);
    }
    __device__ T zoutc(const ZC &, int, int) const { return (T)0; }
    __device__ void xyi_put(int tj, int, int, size_t p, V s) const { xyi_flush(tj, p, s); }
    static constexpr int NF = 1, NB = 1;
    const V *Rpsi, *Rocc;     // chunk's first target / source
    double2 *acc;
    const double *fill;
    __device__ V xyf_load(int item, int, int, int, int, size_t p) const
    {
        const int tj = item / this->ns, si = item % this->ns;
        return cmulc(__ldg(&Rocc[(size_t)si * this->g.N + p]), __ldg(&Rpsi[(size_t)tj * this->g.N + p]));
    }
    __device__ V zmix(int item, int, int x, int y, int z, const V *in) const
    {
        // 1/|k-q+G|^2 (hf2x.cpp:93-104) with the 1/N of the forward transform (TAB_HF)
        const size_t p = (size_t)this->pair_id(item) * this->g.N + this->pidx(x, y, z);
        if constexpr (OpBase<T>::FT) return cscale(in[0], __ldg(this->m.ftab + p));
        else return cscale(in[0], __ldg(this->m.tab + p));
    }
    __device__ void xyi_accum(int tj, int item, int, size_t p, const V *v) const
    {
        const int si = item % this->ns;
        acc_red(acc + (size_t)tj * this->g.N + p, to64(cmul(v[0], __ldg(&Rocc[(size_t)si * this->g.N + p]))), fill[si]);
    }
};

// =================================================================== tc2x ==
template <typename T>
struct OpTC2X : OpBase<T> {
    using V = typename C2<T>::t;
    static constexpr const char *NAME = "tc2x";
    static constexpr unsigned BLI = 0xF, BLO = 0xF;
    static constexpr bool ZSPLIT = false;     // one thread per z-line measured faster here
    static constexpr bool REGACC = true;
    __device__ bool regacc_grid(int) const { return true; }
    __device__ V xyi_term(int, int item, int b, size_t p, const V *v) const
    {
        const size_t N = this->g.N;
        const int si = item % this->ns;
        const V o = b == 0 ? __ldg(&Rocc[(size_t)si * N + p]) : __ldg(&Rgrad[((size_t)si * 3 + (b - 1)) * N + p]);
        return cscale(cmul(v[0], o), (decltype(v[0].x))(b == 0 ? fill[si] : -fill[si]));
    }
    __device__ void xyi_flush(int tj, size_t p, V s) const { acc_red(acc + (size_t)tj * this->g.N + p, to64(s), 1.0); }
    __device__ const V *xyi_operand(int, int b, int si) const
    {
        return b == 0 ? Rocc + (size_t)si * this->g.N : Rgrad + ((size_t)si * 3 + (b - 1)) * this->g.N;
    }
    template <class F> __device__ void xyi_add(int si, int b, const V *v, const V *o, F &&add) const
    {
        add(0, cscale64(cmul(v[0], o[0]), b == 0 ? fill[si] : -fill[si]));
    }
    __device__ const V *xyf_operand(int, int, int si) const { return Rchi + (size_t)si * this->g.N; }
    __device__ V xyf_pair(int tj, int f, size_t p, const V *o) const
    {
        const size_t N = this->g.N;
        return cmulc(o[0], f == 0 ? __ldg(&Rpsi[(size_t)tj * N + p]) : __ldg(&Rgpsi[((size_t)tj * 3 + (f - 1)) * N + p]));
    }
    // coefficient planes: V_2body, du_0, du_1, du_2
    using ZC = typename OpBase<T>::ZC;
    __device__ ZC zctx(int item, int x, int y, int c) const { return this->zctx_base(item, x, y, c, 2); }
    __device__ T zmixc(const ZC &c, int f, int z) const
    {
        if constexpr (OpBase<T>::FT) return this->zpl(c, f, z);
        else if (f == 0) return this->zcol(c, 2, 0, z) * this->invN;
        else return this->zdu(c, 2, 1, f - 1, z);
    }
    __device__ T zoutc(const ZC &c, int o, int z) const { return zmixc(c, o, z); }
    __device__ void xyi_put(int tj, int, int, size_t p, V s) const { xyi_flush(tj, p, s); }
    static constexpr int NF = 4, NB = 4;
    const V *Rpsi, *Rgpsi;        // [nt][N], [nt][3][N]
    const V *Rocc, *Rchi, *Rgrad; // [ns][N], [ns][N], [ns][3][N]
    double2 *acc;
    const double *fill;
    __device__ V xyf_load(int item, int f, int, int, int, size_t p) const
    {
        const size_t N = this->g.N;
        const int tj = item / this->ns, si = item % this->ns;
        const V chi = __ldg(&Rchi[(size_t)si * N + p]);
        const V rhs = f == 0 ? __ldg(&Rpsi[(size_t)tj * N + p]) : __ldg(&Rgpsi[((size_t)tj * 3 + (f - 1)) * N + p]);
        return cmulc(chi, rhs);     // tc2x.cpp:350, :374
    }
    __device__ V zmix(int item, int o, int x, int y, int z, const V *in) const
    {
        using S = decltype(in[0].x);
        if constexpr (OpBase<T>::FT) {
            const size_t p = this->pidx(x, y, z);
            V r = cscale(in[0], this->fco(item, p, o));
            if (o == 0) {
                r = cadd(r, cscale(in[1], this->fco(item, p, 1)));
                r = cadd(r, cscale(in[2], this->fco(item, p, 2)));
                r = cadd(r, cscale(in[3], this->fco(item, p, 3)));
            }
            return r;
        }
        double G[3];
        gvec(this->rc.R, this->g, x, y, z, this->kq_of(item), G);
        const size_t p = this->pidx(x, y, z);
        const double *tab = this->tab_of(item);
        const double u = tab[2 * p + 1] * this->invN;
        if (o == 0) {   // [2a_x] rho V_2body + [2b_x2] sum_d rho_d du_d   (tc2x.cpp:378-386)
            V r = cscale(in[0], (S)(tab[2 * p] * this->invN));
#pragma unroll
            for (int d = 0; d < 3; d++) r = cadd(r, cscale(in[1 + d], (S)(G[d] * u)));
            return r;
        }
        return cscale(in[0], (S)(G[o - 1] * u));   // [2b_x1] rho du_d (tc2x.cpp:354-358)
    }
    __device__ void xyi_accum(int tj, int item, int b, size_t p, const V *v) const
    {
        const size_t N = this->g.N;
        const int si = item % this->ns;
        const V o = b == 0 ? __ldg(&Rocc[(size_t)si * N + p]) : __ldg(&Rgrad[((size_t)si * 3 + (b - 1)) * N + p]);
        acc_red(acc + (size_t)tj * N + p, to64(cmul(v[0], o)), b == 0 ? fill[si] : -fill[si]);
    }
};

// Jastrow tables per (tb, sb): modes select the columns
enum TabMode { TAB_TC2X = 0, TAB_U_SX = 1, TAB_U_SS = 2, TAB_U_QX = 3, TAB_HF = 4 };
// TAB_TC2X : [V_2body(s,s), u(s,s)]                         (tc2x.cpp:266-276)
// TAB_U_SX : [u(G; 0, s), u(G; 1, s)]                        (tc3a3b3b4b6.cpp:208-217)
// TAB_U_SS : [u(G; s, s)]                                    (tc3a3b3b4b6.cpp:679-686)
// TAB_U_QX : [u(G; s, 0), u(G; s, 1)]                        (tc3a2a4b2b5.cpp:244-253)
// TAB_HF   : [1/(N |G|^2), 0 where |G|^2 < 1e-8]             (hf2x.cpp:93-104)
// Points in the order of the grids between the passes (tr: y fastest in a plane).
__device__ __forceinline__ void xyz_tab(const GridDesc &g, int tr, size_t p, int &x, int &y, int &z)
{
    if (tr) {
        y = (int)(p % g.n1);
        x = (int)((p / g.n1) % g.n0);
        z = (int)(p / ((size_t)g.n0 * g.n1));
    } else xyz_of(g, p, x, y, z);
}
// wrap: the pair densities' sphere reaches past the work grid's box
// (workgrid.cuh), so a grid point stands for the image of G under the grid's
// periods that lies in it (the shortest k - q + G); the value is the one the
// caller's grid un has at that component.
struct HFGrid {
    int wrap, un[3];
};
__device__ __forceinline__ double hf_kernel(const double *q, const double *R, const GridDesc &g, const HFGrid &hg, int x, int y,
                                            int z, double invN)
{
    int m[3] = {miller(x, g.n0), miller(y, g.n1), miller(z, g.n2)};
    if (hg.wrap) {
        double best = 1e300;
        int b[3] = {0, 0, 0};
        for (int i = 0; i < 27; i++) {
            const int s[3] = {m[0] + (i % 3 - 1) * g.n0, m[1] + (i / 3 % 3 - 1) * g.n1, m[2] + (i / 9 - 1) * g.n2};
            double v = 0;
#pragma unroll
            for (int d = 0; d < 3; d++) {
                const double c = q[d] + R[d] * s[0] + R[3 + d] * s[1] + R[6 + d] * s[2];
                v += c * c;
            }
            if (v < best) {
                best = v;
                for (int d = 0; d < 3; d++) b[d] = s[d];
            }
        }
        for (int d = 0; d < 3; d++) {
            int u = b[d] % hg.un[d];
            if (u < 0) u += hg.un[d];
            m[d] = miller(u, hg.un[d]);
        }
    }
    double t = 0;
#pragma unroll
    for (int d = 0; d < 3; d++) {
        const double c = q[d] + R[d] * m[0] + R[3 + d] * m[1] + R[6 + d] * m[2];
        t += c * c;
    }
    return t < 1e-8 ? 0.0 : invN / t;
}
static __global__ void k_tables(GridDesc g, RecipC rc, Jastrow J, int mode, int tr, HFGrid hg, int s, int npair,
                                const double *kq, double invN, double *tab)
{
    const int ntab = mode == TAB_U_SS || mode == TAB_HF ? 1 : 2;
    const size_t total = (size_t)npair * g.N;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int pr = (int)(i / g.N);
        const size_t p = i % g.N;
        int x, y, z;
        xyz_tab(g, tr, p, x, y, z);
        double G[3];
        gvec(rc.R, g, x, y, z, kq + 3 * pr, G);
        double *o = tab + i * ntab;
        if (mode == TAB_HF) o[0] = hf_kernel(kq + 3 * pr, rc.R, g, hg, x, y, z, invN);
        else if (mode == TAB_TC2X) { o[0] = J.tc2body(G, s, s); o[1] = J.uk(G, s, s); }
        else if (mode == TAB_U_SX) { o[0] = J.uk(G, 0, s); o[1] = J.uk(G, 1, s); }
        else if (mode == TAB_U_SS) { o[0] = J.uk(G, s, s); }
        else { o[0] = J.uk(G, s, 0); o[1] = J.uk(G, s, 1); }
    }
}

// FP32 coefficient tables of the mixed path, evaluated in FP64 and rounded
// once; G = k - q + G_p, all include the 1/N of the forward transform; a pair's
// planes of N points each:
//   TAB_TC2X : V_2body(s,s), G_0 u, G_1 u, G_2 u     with u = u(G; s, s)
//   TAB_U_SX : G_d u(G; x, s), plane 3 x + d (3 planes: x = s alone)
//   TAB_U_SS : G_d u(G; s, s)
//   TAB_U_QX : G_d u(G; s, x), plane 3 x + d (3 planes: x = s alone)
//   TAB_HF   : 1 / |G|^2
static __global__ void k_ftables(GridDesc g, RecipC rc, Jastrow J, int mode, int tr, HFGrid hg, int s, int nrec, int npair,
                                 const double *kq, double invN, float *tab)
{
    const size_t total = (size_t)npair * g.N;
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < total; i += (size_t)gridDim.x * blockDim.x) {
        const int pr = (int)(i / g.N);
        const size_t p = i % g.N;
        int x, y, z;
        xyz_tab(g, tr, p, x, y, z);
        float *o = tab + (size_t)pr * nrec * g.N + p;
        if (mode == TAB_HF) {
            o[0] = (float)hf_kernel(kq + 3 * pr, rc.R, g, hg, x, y, z, invN);
            continue;
        }
        double G[3];
        gvec(rc.R, g, x, y, z, kq + 3 * pr, G);
        int r0 = 0;
        if (mode == TAB_TC2X) {
            o[0] = (float)(J.tc2body(G, s, s) * invN);
            r0 = 1;
        }
        const int nx = (nrec - r0) / 3;
        for (int x2 = 0; x2 < nx; x2++) {
            const int xr = nx == 1 ? s : x2;
            const double u = (mode == TAB_U_SX ? J.uk(G, xr, s) : (mode == TAB_U_QX ? J.uk(G, s, xr) : J.uk(G, s, s))) * invN;
            for (int d = 0; d < 3; d++) o[(size_t)(r0 + 3 * x2 + d) * g.N] = (float)(G[d] * u);
        }
    }
}

// ======================================================= tc3a3b3b4b6 ops ==
// stage A: first q loop (tc3a3b3b4b6.cpp:192-368).
// EQ: u(G; 0, s) == u(G; 1, s) (same Jastrow A, F for both spins of x2), so
// the spin sum of the 3b6 chain collapses by linearity,
//   sum_x du_d FFT[n_x IFFT[phiphi du_d]] = du_d FFT[(n_0 + n_1) IFFT[phiphi du_d]],
// and only three P grids (x = s) are needed instead of six.
template <typename T, bool EQ = false>
struct OpTC3A : OpBase<T> {
    using V = typename C2<T>::t;
    static constexpr const char *NAME = "3a3b6A";
    static constexpr int NX = EQ ? 1 : 2;     // spin branches of x2 carried
    static constexpr int NF = 4, NB = 1 + 3 * NX;
    static constexpr unsigned BLI = 0xF, BLO = (1u << NB) - 1;
    static constexpr bool REFWD = true;
    static constexpr bool ZSPLIT = false;    // one thread per z-line measured faster here
    // one-thread and lane-pair forms: accumulation through xyi_accum (FP64 red.add per
    // source), so that the prefetching XYI kernel can transform the re-forwarded planes
    // in place
    static constexpr bool REGACC = false, BOUTER = true;
    __device__ bool regacc_grid(int b) const { return b == 0 || EQ || (b - 1) / 3 == s; }
    __device__ V xyi_term(int, int item, int b, size_t p, const V *v) const
    {
        const int si = item % this->ns;
        const V t = cmul(v[0], __ldg(&Rocc[(size_t)si * this->g.N + p]));
        return b == 0 ? cscale(t, (decltype(t.x))(fill[si] * b3)) : t;
    }
    __device__ void xyi_flush_b(int tj, int b, size_t p, V sum) const
    {
        const size_t N = this->g.N;
        if (b == 0) acc_red(acc + (size_t)tj * N + p, to64(sum), 1.0);
        else acc_red(qsum + ((size_t)tj * 3 + (b - 1) % 3) * N + p, to64(sum), 1.0);
    }
    const V *Rpsi, *Rocc, *Rchi;  // [nt][N], [ns][N]
    const V *dnu;                 // [3][N] of the targets' spin
    const V *densT;               // [2][N] density (EQ: [0] = n_0 + n_1), compute precision
    double2 *acc, *qsum;          // [nt][N], [nt][3][N]
    const double *fill;
    V *tmp2;                      // [items][3 NX][N]
    int s;
    double b3;
    __device__ V xyf_load(int item, int f, int, int, int, size_t p) const
    {
        const size_t N = this->g.N;
        const int tj = item / this->ns, si = item % this->ns;
        const V chi = __ldg(&Rchi[(size_t)si * N + p]);
        V rhs = __ldg(&Rpsi[(size_t)tj * N + p]);
        if (f > 0) rhs = cmul(__ldg(&dnu[(size_t)(f - 1) * N + p]), rhs);   // dnu_phi (:236)
        return cmulc(chi, rhs);
    }
    __device__ V zmix(int item, int o, int x, int y, int z, const V *in) const
    {
        using S = decltype(in[0].x);
        if constexpr (OpBase<T>::FT) {
            const size_t p = this->pidx(x, y, z);
            if (o == 0) {
                const int r0 = EQ ? 0 : 3 * s;
                V r = cscale(in[1], this->fco(item, p, r0));
                r = cadd(r, cscale(in[2], this->fco(item, p, r0 + 1)));
                return cadd(r, cscale(in[3], this->fco(item, p, r0 + 2)));
            }
            return cscale(in[0], (float)fill[item % this->ns] * this->fco(item, p, o - 1));   // plane 3 xs + d
        }
        double G[3];
        gvec(this->rc.R, this->g, x, y, z, this->kq_of(item), G);
        const size_t p = this->pidx(x, y, z);
        const double *tab = this->tab_of(item) + 2 * p;
        if (o == 0) {   // [3b3] sum_d du[s]_d FFT(dnu_phi_d conj chi) (:286-295)
            const double u = tab[s] * this->invN;
            V r = cscale(in[1], (S)(G[0] * u));
            r = cadd(r, cscale(in[2], (S)(G[1] * u)));
            return cadd(r, cscale(in[3], (S)(G[2] * u)));
        }
        const int xs = EQ ? s : (o - 1) / 3, d = (o - 1) % 3;   // phiphi f du[xs]_d (:306-314)
        const double f = fill[item % this->ns];
        return cscale(in[0], (S)(f * G[d] * tab[xs] * this->invN));
    }
    __device__ void xyi_accum(int tj, int item, int b, size_t p, const V *v) const
    {
        const size_t N = this->g.N;
        const int si = item % this->ns;
        const V phq = __ldg(&Rocc[(size_t)si * N + p]);
        if (b == 0) {
            acc_red(acc + (size_t)tj * N + p, to64(cmul(v[0], phq)), fill[si] * b3);
        } else {
            const int xs = EQ ? s : (b - 1) / 3, d = (b - 1) % 3;
            if (xs == s) acc_red(qsum + ((size_t)tj * 3 + d) * N + p, to64(cmul(v[0], phq)), 1.0);
        }
    }
    __device__ bool refwd_want(int b) const { return b > 0; }
    static constexpr int NRW = NX;
    __device__ const V *refwd_dens(int xs) const { return densT + (size_t)xs * this->g.N; }
    __device__ V refwd_mul(int, V v, V n) const { return cmul(v, n); }   // orbital * n_s2 (:332)
    __device__ V refwd_load(int, int item, int b, size_t p, V v) const
    {
        return refwd_mul(item, v, __ldg(refwd_dens(EQ ? 0 : (b - 1) / 3) + p));
    }
    // one sum per output: b3 f v phi_q (b = 0), v phi_q of the branch x = s
    __device__ const V *xyi_operand(int, int b, int si) const
    {
        return regacc_grid(b) ? Rocc + (size_t)si * this->g.N : nullptr;
    }
    template <class F> __device__ void xyi_add(int si, int b, const V *v, const V *o, F &&add) const
    {
        const V t = cmul(v[0], o[0]);
        if (regacc_grid(b)) add(0, b == 0 ? cscale64(t, fill[si] * b3) : t);
    }
    __device__ void xyi_put(int tj, int b, int, size_t p, V sum) const
    {
        if (regacc_grid(b)) xyi_flush_b(tj, b, p, sum);
    }
    __device__ const V *xyf_operand(int, int, int si) const { return Rchi + (size_t)si * this->g.N; }
    __device__ V xyf_pair(int tj, int f, size_t p, const V *o) const
    {
        V rhs = __ldg(&Rpsi[(size_t)tj * this->g.N + p]);
        if (f > 0) rhs = cmul(__ldg(&dnu[(size_t)(f - 1) * this->g.N + p]), rhs);
        return cmulc(o[0], rhs);
    }
    static constexpr int ZM0 = 1;
    using ZC = typename OpBase<T>::ZC;
    __device__ ZC zctx(int item, int x, int y, int c) const
    {
        ZC z = this->zctx_base(item, x, y, c, 2);
        z.f = (T)fill[item % this->ns];
        return z;
    }
    __device__ T branch_du(const ZC &c, int xs, int d, int z) const
    {
        if constexpr (OpBase<T>::FT) return this->zpl(c, (EQ ? 0 : 3 * xs) + d, z);
        else return this->zdu(c, 2, xs, d, z);
    }
    __device__ T zmixc(const ZC &c, int f, int z) const { return branch_du(c, s, f - 1, z); }
    __device__ T zoutc(const ZC &c, int o, int z) const { return c.f * branch_du(c, EQ ? s : (o - 1) / 3, (o - 1) % 3, z); }
    __device__ V *refwd_grid(int item, int b) const { return tmp2 + ((size_t)item * 3 * NX + (b - 1)) * this->g.N; }
};

// stage B: [3b6] sum_{s2,d} FFT(.) du[s2]_d -> IFFT x phi_q (:333-348)
template <typename T, bool EQ = false>
struct OpTC3B : OpBase<T> {
    using V = typename C2<T>::t;
    static constexpr const char *NAME = "3b6B";
    static constexpr int NX = EQ ? 1 : 2;
    static constexpr int NF = 3 * NX, NB = 1;
    static constexpr unsigned BLI = (1u << NF) - 1, BLO = 1;
    static constexpr bool REGACC = true;
    __device__ bool regacc_grid(int) const { return true; }
    __device__ V xyi_term(int, int item, int, size_t p, const V *v) const
    {
        const int si = item % this->ns;
        return cscale(cmul(v[0], __ldg(&Rocc[(size_t)si * this->g.N + p])), (decltype(v[0].x))b6);
    }
    __device__ void xyi_flush(int tj, size_t p, V s) const { acc_red(acc + (size_t)tj * this->g.N + p, to64(s), 1.0); }
    __device__ const V *xyi_operand(int, int, int si) const { return Rocc + (size_t)si * this->g.N; }
    template <class F> __device__ void xyi_add(int si, int, const V *v, const V *o, F &&add) const
    {
        add(0, cmul(v[0], o[0]));
    }
    // in the coefficient planes / columns of tc3a3b3b4b6's tables, or after tc2x's
    // V_2body plane (c0 = 1) and in its u column (col = 1) in the shared pass
    int c0 = 0, col = -1;
    static constexpr int NSO = 0;             // no forward pass
    using ZC = typename OpBase<T>::ZC;
    __device__ ZC zctx(int item, int x, int y, int c) const { return this->zctx_base(item, x, y, c, 2); }
    __device__ T zmixc(const ZC &c, int f, int z) const
    {
        if constexpr (OpBase<T>::FT) return this->zpl(c, c0 + f, z);
        else return this->zdu(c, 2, col >= 0 ? col : (EQ ? s : f / 3), f % 3, z);
    }
    __device__ T zoutc(const ZC &, int, int) const { return (T)0; }
    __device__ void xyi_put(int tj, int, int, size_t p, V s) const { acc_red(acc + (size_t)tj * this->g.N + p, to64(s), b6); }
    const V *Rocc;
    double2 *acc;
    V *tmp2;
    double b6;
    int s;
    __device__ V *zin_grid(int item, int f) const { return tmp2 + ((size_t)item * NF + f) * this->g.N; }
    __device__ V zmix(int item, int, int x, int y, int z, const V *in) const
    {
        using S = decltype(in[0].x);
        if constexpr (OpBase<T>::FT) {
            const size_t p = this->pidx(x, y, z);
            V r = czero<V>();
#pragma unroll
            for (int xs = 0; xs < NX; xs++) {
                r = cadd(r, cscale(in[3 * xs], this->fco(item, p, 3 * xs)));
                r = cadd(r, cscale(in[3 * xs + 1], this->fco(item, p, 3 * xs + 1)));
                r = cadd(r, cscale(in[3 * xs + 2], this->fco(item, p, 3 * xs + 2)));
            }
            return r;
        }
        double G[3];
        gvec(this->rc.R, this->g, x, y, z, this->kq_of(item), G);
        const size_t p = this->pidx(x, y, z);
        const double *tab = this->tab_of(item) + 2 * p;
        V r = czero<V>();
#pragma unroll
        for (int xs = 0; xs < NX; xs++) {
            const double u = tab[EQ ? s : xs] * this->invN;
#pragma unroll
            for (int d = 0; d < 3; d++) r = cadd(r, cscale(in[3 * xs + d], (S)(G[d] * u)));
        }
        return r;
    }
    __device__ void xyi_accum(int tj, int item, int, size_t p, const V *v) const
    {
        const int si = item % this->ns;
        acc_red(acc + (size_t)tj * this->g.N + p, to64(cmul(v[0], __ldg(&Rocc[(size_t)si * this->g.N + p]))), b6);
    }
};

// stage C: [3b4] second q loop (:664-767)
template <typename T>
struct OpTC3C : OpBase<T> {
    using V = typename C2<T>::t;
    static constexpr const char *NAME = "3b4C";
    static constexpr bool REGACC = true;
    __device__ bool regacc_grid(int) const { return true; }
    __device__ V xyi_term(int, int item, int, size_t p, const V *v) const
    {
        const int si = item % this->ns;
        return cscale(cmul(v[0], __ldg(&Rocc[(size_t)si * this->g.N + p])), (decltype(v[0].x))(b4 * fill[si]));
    }
    __device__ void xyi_flush(int tj, size_t p, V s) const { acc_red(acc + (size_t)tj * this->g.N + p, to64(s), 1.0); }
    __device__ const V *xyi_operand(int, int, int si) const { return Rocc + (size_t)si * this->g.N; }
    template <class F> __device__ void xyi_add(int si, int, const V *v, const V *o, F &&add) const
    {
        add(0, cscale64(cmul(v[0], o[0]), b4 * fill[si]));
    }
    __device__ const V *xyf_operand(int, int, int si) const { return Rchi + (size_t)si * this->g.N; }
    __device__ V xyf_pair(int tj, int f, size_t p, const V *o) const
    {
        return cmulc(o[0], from64<V>(__ldg(&qsum[((size_t)tj * 3 + f) * this->g.N + p])));
    }
    using ZC = typename OpBase<T>::ZC;
    __device__ ZC zctx(int item, int x, int y, int c) const { return this->zctx_base(item, x, y, c, 1); }
    __device__ T zmixc(const ZC &c, int f, int z) const
    {
        if constexpr (OpBase<T>::FT) return this->zpl(c, f, z);
        else return this->zdu(c, 1, 0, f, z);
    }
    __device__ T zoutc(const ZC &, int, int) const { return (T)0; }
    __device__ void xyi_put(int tj, int, int, size_t p, V s) const { xyi_flush(tj, p, s); }
    static constexpr int NF = 3, NB = 1;
    static constexpr unsigned BLI = 7, BLO = 1;
    const V *Rocc, *Rchi;
    const double2 *qsum;      // [nt][3][N]
    double2 *acc;
    const double *fill;
    double b4;
    __device__ V xyf_load(int item, int f, int, int, int, size_t p) const
    {
        const size_t N = this->g.N;
        const int tj = item / this->ns, si = item % this->ns;
        return cmulc(__ldg(&Rchi[(size_t)si * N + p]), from64<V>(__ldg(&qsum[((size_t)tj * 3 + f) * N + p])));
    }
    __device__ V zmix(int item, int, int x, int y, int z, const V *in) const
    {
        using S = decltype(in[0].x);
        if constexpr (OpBase<T>::FT) {
            const size_t p = this->pidx(x, y, z);
            V r = cscale(in[0], this->fco(item, p, 0));
            r = cadd(r, cscale(in[1], this->fco(item, p, 1)));
            return cadd(r, cscale(in[2], this->fco(item, p, 2)));
        }
        double G[3];
        gvec(this->rc.R, this->g, x, y, z, this->kq_of(item), G);
        const size_t p = this->pidx(x, y, z);
        const double u = this->tab_of(item)[p] * this->invN;
        V r = cscale(in[0], (S)(G[0] * u));
        r = cadd(r, cscale(in[1], (S)(G[1] * u)));
        return cadd(r, cscale(in[2], (S)(G[2] * u)));
    }
    __device__ void xyi_accum(int tj, int item, int, size_t p, const V *v) const
    {
        const int si = item % this->ns;
        acc_red(acc + (size_t)tj * this->g.N + p, to64(cmul(v[0], __ldg(&Rocc[(size_t)si * this->g.N + p]))), b4 * fill[si]);
    }
};

// 3b3 (tc3a3b3b4b6.cpp:284-302), 3b4 (:651-770) and 3b5 (tc3a2a4b2b5.cpp:
// 882-894) each transform three grids, contract them with du_d(G) =
// (k - q + G)_d u(G; s, s) and multiply the inverse transform by phi_q f_q:
// by linearity one transform of the sum of their scaled inputs,
//   in_d = conj(chi_q) (b3 dnu_d psi_k + b4 qsum_d[k]) + b5 Bt_d[q] psi_k,
// gives all three (b5 = 0 without tc3a2a4b2b5).  Runs in the second q loop,
// after the first has completed qsum.
template <typename T>
struct OpTC3X : OpBase<T> {
    using V = typename C2<T>::t;
    static constexpr const char *NAME = "3bX";
    static constexpr int NF = 3, NB = 1;
    static constexpr unsigned BLI = 7, BLO = 1;
    static constexpr bool REGACC = true;
    __device__ bool regacc_grid(int) const { return true; }
    const V *Rpsi, *Rocc, *Rchi;  // [nt][N], [ns][N], [ns][N]
    const V *W;                   // [nt][3][N] per-target part b3 dnu_d psi + b4 qsum_d (k_w3x)
    const V *Bt;                  // [ns][3][N] or null (b5 = 0)
    double2 *acc;
    const double *fill;
    double b5;
    __device__ V xyf_load(int item, int f, int, int, int, size_t p) const
    {
        using S = decltype(V{}.x);
        const size_t N = this->g.N;
        const int tj = item / this->ns, si = item % this->ns;
        V r = cmulc(__ldg(&Rchi[(size_t)si * N + p]), __ldg(&W[((size_t)tj * 3 + f) * N + p]));
        if (Bt) r = cadd(r, cscale(cmul(__ldg(&Bt[((size_t)si * 3 + f) * N + p]), __ldg(&Rpsi[(size_t)tj * N + p])), (S)b5));
        return r;
    }
    __device__ V zmix(int item, int, int x, int y, int z, const V *in) const
    {
        using S = decltype(in[0].x);
        if constexpr (OpBase<T>::FT) {
            const size_t p = this->pidx(x, y, z);
            V r = cscale(in[0], this->fco(item, p, 0));
            r = cadd(r, cscale(in[1], this->fco(item, p, 1)));
            return cadd(r, cscale(in[2], this->fco(item, p, 2)));
        }
        double G[3];
        gvec(this->rc.R, this->g, x, y, z, this->kq_of(item), G);
        const size_t p = this->pidx(x, y, z);
        const double u = this->tab_of(item)[p] * this->invN;
        V r = cscale(in[0], (S)(G[0] * u));
        r = cadd(r, cscale(in[1], (S)(G[1] * u)));
        return cadd(r, cscale(in[2], (S)(G[2] * u)));
    }
    __device__ V xyi_term(int, int item, int, size_t p, const V *v) const
    {
        const int si = item % this->ns;
        return cscale(cmul(v[0], __ldg(&Rocc[(size_t)si * this->g.N + p])), (decltype(v[0].x))fill[si]);
    }
    __device__ void xyi_flush(int tj, size_t p, V s) const { acc_red(acc + (size_t)tj * this->g.N + p, to64(s), 1.0); }
    __device__ const V *xyi_operand(int, int, int si) const { return Rocc + (size_t)si * this->g.N; }
    template <class F> __device__ void xyi_add(int si, int, const V *v, const V *o, F &&add) const
    {
        add(0, cscale64(cmul(v[0], o[0]), fill[si]));
    }
    static constexpr int NSO = 2;
    __device__ const V *xyf_operand(int k, int f, int si) const
    {
        return k == 0 ? Rchi + (size_t)si * this->g.N : (Bt ? Bt + ((size_t)si * 3 + f) * this->g.N : nullptr);
    }
    __device__ V xyf_pair(int tj, int f, size_t p, const V *o) const
    {
        const size_t N = this->g.N;
        V r = cmulc(o[0], __ldg(&W[((size_t)tj * 3 + f) * N + p]));
        if (Bt) r = cadd(r, cscale(cmul(o[1], __ldg(&Rpsi[(size_t)tj * N + p])), (T)b5));
        return r;
    }
    using ZC = typename OpBase<T>::ZC;
    __device__ ZC zctx(int item, int x, int y, int c) const { return this->zctx_base(item, x, y, c, 1); }
    __device__ T zmixc(const ZC &c, int f, int z) const
    {
        if constexpr (OpBase<T>::FT) return this->zpl(c, f, z);
        else return this->zdu(c, 1, 0, f, z);
    }
    __device__ T zoutc(const ZC &, int, int) const { return (T)0; }
    __device__ void xyi_put(int tj, int, int, size_t p, V s) const { xyi_flush(tj, p, s); }
    __device__ void xyi_accum(int tj, int item, int, size_t p, const V *v) const
    {
        const int si = item % this->ns;
        acc_red(acc + (size_t)tj * this->g.N + p, to64(cmul(v[0], __ldg(&Rocc[(size_t)si * this->g.N + p]))), fill[si]);
    }
};

// ======================================================= tc3a2a4b2b5 ops ==
// occupied-pair stage (tc3a2a4b2b5.cpp:210-443): targets (q2, i2), sources (q1, i1).
// EQ: u(G; sq, 0) == u(G; sq, 1), so both branches x2 = 0, 1 give the same
// orbital grids; one branch is transformed and its 3a2 contribution is
// added to both spin slots (twice into slot 0 when unpolarised).
template <typename T, bool BITC, bool EQ = false>
struct OpQP : OpBase<T> {
    using V = typename C2<T>::t;
    static constexpr const char *NAME = "qp";
    static constexpr int NX = EQ ? 1 : 2;
    static constexpr int NF = BITC ? 2 : 1, NB = (BITC ? 6 : 3) * NX, GS = BITC ? 2 : 1;
    static constexpr unsigned BLI = (1u << NF) - 1, BLO = (1u << NB) - 1;
    const V *Rq2, *Rq2c;          // targets phi_q2(r), chi_q2(r)  [nt][N]
    const V *Rocc, *Rchi;         // sources phi_q1, chi_q1        [ns][N]
    double2 *acc;                 // [nt][nacc][N]: 3a2[nspin], 3a4[3], 3b5[3]
    const double *fill;           // sources
    int nacc, nspin, sq;
    __device__ V xyf_load(int item, int f, int, int, int, size_t p) const
    {
        const size_t N = this->g.N;
        const int tj = item / this->ns, si = item % this->ns;
        if (f == 0) return cmulc(__ldg(&Rchi[(size_t)si * N + p]), __ldg(&Rq2[(size_t)tj * N + p]));   // (:359)
        return cmulc(__ldg(&Rocc[(size_t)si * N + p]), __ldg(&Rq2c[(size_t)tj * N + p]));              // (:365)
    }
    __device__ V zmix(int item, int o, int x, int y, int z, const V *in) const
    {
        using S = decltype(in[0].x);
        if constexpr (OpBase<T>::FT) {
            int xs, d, w;
            if (BITC) { w = o & 1; xs = (o >> 1) / 3; d = (o >> 1) % 3; }
            else { w = 0; xs = o / 3; d = o % 3; }
            return cscale(in[w], this->fco(item, this->pidx(x, y, z), (EQ ? 0 : 3 * xs) + d));
        }
        double G[3];
        gvec(this->rc.R, this->g, x, y, z, this->kq_of(item), G);
        const size_t p = this->pidx(x, y, z);
        const double *tab = this->tab_of(item) + 2 * p;
        int xs, d, w;
        if (BITC) { w = o & 1; xs = (o >> 1) / 3; d = (o >> 1) % 3; }
        else { w = 0; xs = o / 3; d = o % 3; }
        if (EQ) xs = sq;
        return cscale(in[w], (S)(G[d] * tab[xs] * this->invN));   // du[x]_d * phiphi (:378, :385)
    }
    // a group's sums: 0 = 3a2 of its branch x2, 1 = 3a4_d, 2 = 3b5_d (x2 = sq)
    static constexpr int NACC = BITC ? 3 : 2;
    __device__ void branch(int b, int &xs, int &d) const
    {
        if (BITC) { xs = (b >> 1) / 3; d = (b >> 1) % 3; }
        else { xs = b / 3; d = b % 3; }
        if (EQ) xs = sq;
    }
    static constexpr int NOPS = BITC ? 2 : 1;
    __device__ const V *xyi_operand(int k, int b, int si) const
    {
        int xs, d;
        branch(b, xs, d);
        return xs == sq ? (k == 0 ? Rocc : Rchi) + (size_t)si * this->g.N : nullptr;
    }
    template <class F> __device__ void xyi_add(int si, int b, const V *v, const V *o, F &&add) const
    {
        const double f1 = fill[si];
        int xs, d;
        branch(b, xs, d);
        const V o1 = v[0];
        if constexpr (BITC) add(0, cscale64(cmulc(v[1], o1), -f1));                          // (:392-394)
        else add(0, cscale64(V{o1.x * o1.x + o1.y * o1.y, (T)0}, -f1));                      // (:404-406)
        if (xs == sq) {
            add(1, cscale64(cmul(o1, o[0]), f1));
            if constexpr (BITC) add(2, cscale64(cconj(cmul(v[1], o[1])), -f1));              // (:428-430)
        }
    }
    static constexpr int ZK = NF, ZMO = -1;
    __device__ int zsrc(int o) const { return BITC ? o & 1 : 0; }
    using ZC = typename OpBase<T>::ZC;
    __device__ ZC zctx(int item, int x, int y, int c) const { return this->zctx_base(item, x, y, c, 2); }
    __device__ T zmixc(const ZC &, int, int) const { return (T)0; }
    __device__ T zoutc(const ZC &c, int o, int z) const
    {
        const int w = BITC ? o >> 1 : o, xs = EQ ? sq : w / 3, d = w % 3;
        if constexpr (OpBase<T>::FT) return this->zpl(c, (EQ ? 0 : 3 * xs) + d, z);
        else return this->zdu(c, 2, xs, d, z);
    }
    __device__ const V *xyf_operand(int, int f, int si) const { return (f == 0 ? Rchi : Rocc) + (size_t)si * this->g.N; }
    __device__ V xyf_pair(int tj, int f, size_t p, const V *o) const
    {
        return cmulc(o[0], __ldg(&(f == 0 ? Rq2 : Rq2c)[(size_t)tj * this->g.N + p]));
    }
    __device__ void xyi_put(int tj, int b, int slot, size_t p, V sum) const
    {
        const size_t N = this->g.N;
        double2 *A = acc + (size_t)tj * nacc * N + p;
        int xs, d;
        branch(b, xs, d);
        if (slot == 0) {
            // EQ: one branch stands for both, twice into slot 0 (unpolarised) or into 0 and 1
            if (EQ && nspin == 1) acc_red(A, to64(sum), 2.0);
            else if (EQ) { acc_red(A, to64(sum), 1.0); acc_red(A + N, to64(sum), 1.0); }
            else acc_red(A + (size_t)(nspin == 1 ? 0 : xs) * N, to64(sum), 1.0);
        } else if (xs == sq) {
            acc_red(A + (size_t)(nspin + (slot == 2 ? 3 : 0) + d) * N, to64(sum), 1.0);
        }
    }
    __device__ void xyi_accum(int tj, int item, int b, size_t p, const V *v) const
    {
        const size_t N = this->g.N;
        const int si = item % this->ns;
        const double f1 = fill[si];
        int xs, d;
        if (BITC) { xs = (b >> 1) / 3; d = (b >> 1) % 3; }
        else { xs = b / 3; d = b % 3; }
        if (EQ) xs = sq;
        double2 *A = acc + (size_t)tj * nacc * N;
        const double2 o1 = to64(v[0]);
        const double2 c3a2 = BITC ? cmulc(to64(v[1]), o1) : double2{o1.x * o1.x + o1.y * o1.y, 0.0};
        if (EQ) {
            // both x2 branches: slot 0 twice (unpolarised) or slots 0 and 1
            if (nspin == 1) acc_red(A + p, c3a2, -2.0 * f1);
            else { acc_red(A + p, c3a2, -f1); acc_red(A + (size_t)N + p, c3a2, -f1); }
        } else {
            const int xr = nspin == 1 ? 0 : xs;
            acc_red(A + (size_t)xr * N + p, c3a2, -f1);   // (:392-394 BITC, :404-406 TC)
        }
        if (xs == sq) {
            acc_red(A + (size_t)(nspin + d) * N + p, to64(cmul(v[0], __ldg(&Rocc[(size_t)si * N + p]))), f1);
            if (BITC) {
                const double2 cc = to64(cmul(cconj(v[BITC ? 1 : 0]), cconj(__ldg(&Rchi[(size_t)si * N + p]))));
                acc_red(A + (size_t)(nspin + 3 + d) * N + p, cc, -f1);               // (:428-430)
            }
        }
    }
};

// ----------------------------------------- tc2x fused with tc3a3b3b4b6 --
// tc2x and the first q loop of tc3a3b3b4b6 run over the same (target kj,
// source qi) pairs with the same pair density rho = conj(chi_qi) psi_kj.  With
// equal Jastrow channels for the targets' spin the transforms
// w_d = IFFT[rho G_d u(G; s, s)] are tc2x's 2b_x1 grids (tc2x.cpp:353-369) and,
// times the filling, 3a3b6A's outputs 1-3 (tc3a3b3b4b6.cpp:305-349).  OpTC2X3
// is tc2x with those three outputs also summed into qsum_d (3a3 / 3b4) and
// re-forwarded times the density (3b6, for OpTC3B), and with band != 0 also
// the 3a4 band part of tc3a2a4b2b5.  It reads tc2x's coefficient tables
// (TAB_TC2X: V_2body / N and G_d u(s, s) / N), which equal 3a3b6A's for equal
// channels.  The remaining parts that end in sum_d du_d(G) FFT[.] times phi_q
// (3b3, 3b4, 3b5) run as one transform in OpTC3X.
template <typename T>
struct OpTC2X3 : OpTC2X<T> {
    using V = typename C2<T>::t;
    static constexpr const char *NAME = "2x3A";
    static constexpr bool REFWD = true;
    static constexpr bool RACC_EXTRA = true;
    const V *densT;               // [N] n_0 + n_1 (compute precision)
    double2 *qsum;                // [nt][3][N]
    V *tmp2;                      // [items][3][N] re-forwarded grids
    // band part of tc3a2a4b2b5 (band != 0): its outputs 0-2 are f a4 w_d too
    // (tc3a2a4b2b5.cpp:867-875), summed times the rotated intermediate Qt_d
    const V *Qt;                  // [ns][3][N]
    double2 *acc3;                // [nt][N] H3 accumulator
    double fa4;
    int band;
    __device__ bool refwd_want(int b) const { return b > 0; }
    static constexpr int NRW = 1;
    __device__ const V *refwd_dens(int) const { return densT; }
    __device__ V refwd_mul(int item, V v, V n) const
    {
        return cscale(cmul(v, n), (decltype(v.x))this->fill[item % this->ns]);   // f orbital * n (:332)
    }
    __device__ V refwd_load(int, int item, int, size_t p, V v) const { return refwd_mul(item, v, __ldg(densT + p)); }
    __device__ V *refwd_grid(int item, int b) const { return tmp2 + ((size_t)item * 3 + (b - 1)) * this->g.N; }
    // qsum_d += f w_d phi_q (:305-328); tc2x's own sum goes through the registers
    __device__ void xyi_extra(int tj, int item, int b, size_t p, const V *v) const
    {
        if (b == 0) return;
        const size_t N = this->g.N;
        const int si = item % this->ns;
        acc_red(qsum + ((size_t)tj * 3 + (b - 1)) * N + p, to64(cmul(v[0], __ldg(&this->Rocc[(size_t)si * N + p]))),
                this->fill[si]);
        if (band)
            acc_red(acc3 + (size_t)tj * N + p, to64(cmul(__ldg(&Qt[((size_t)si * 3 + (b - 1)) * N + p]), v[0])),
                    this->fill[si] * fa4);
    }
    __device__ void xyi_accum(int tj, int item, int b, size_t p, const V *v) const
    {
        OpTC2X<T>::xyi_accum(tj, item, b, p, v);
        xyi_extra(tj, item, b, p, v);
    }
    // an output's sums: 0 = tc2x's, 1 = qsum_d, 2 = the band part (the last two for b > 0)
    static constexpr int NACC = 3;
    static constexpr int NOPS = 3;           // phi_q, grad_d phi_q, Q_d
    __device__ const V *xyi_operand(int k, int b, int si) const
    {
        const size_t N = this->g.N;
        if (k == 0) return this->Rocc + (size_t)si * N;
        if (b == 0) return nullptr;
        if (k == 1) return this->Rgrad + ((size_t)si * 3 + (b - 1)) * N;
        return band ? Qt + ((size_t)si * 3 + (b - 1)) * N : nullptr;
    }
    template <class F> __device__ void xyi_add(int si, int b, const V *v, const V *o, F &&add) const
    {
        const V w = cscale64(v[0], this->fill[si]);
        if (b == 0) {
            add(0, cmul(w, o[0]));
            return;
        }
        add(0, cscale(cmul(w, o[1]), (T)-1));
        add(1, cmul(w, o[0]));
        if (band) add(2, cmul(w, o[2]));
    }
    __device__ void xyi_put(int tj, int b, int slot, size_t p, V sum) const
    {
        const size_t N = this->g.N;
        if (slot == 0) acc_red(this->acc + (size_t)tj * N + p, to64(sum), 1.0);
        else if (b == 0) return;
        else if (slot == 1) acc_red(qsum + ((size_t)tj * 3 + (b - 1)) * N + p, to64(sum), 1.0);
        else if (band) acc_red(acc3 + (size_t)tj * N + p, to64(sum), fa4);
    }
};

// forward transform of pair products (3a2 divergence correction, :544-550)
template <typename T>
struct OpPairFwd : OpBase<T> {
    using V = typename C2<T>::t;
    static constexpr const char *NAME = "pairfwd";
    static constexpr int NF = 2, NB = 2;
    static constexpr bool ZINV = false;
    static constexpr int ZK = 2, ZMO = -1;
    __device__ int zsrc(int o) const { return o; }
    static constexpr int NSO = 0;
    using ZC = typename OpBase<T>::ZC;
    __device__ ZC zctx(int, int, int, int) const { return ZC{}; }
    __device__ T zmixc(const ZC &, int, int) const { return (T)0; }
    __device__ T zoutc(const ZC &, int, int) const { return (T)this->invN; }
    const V *A0, *B0, *A1, *B1;   // item i: conj(A0_i) B0_i, conj(A1_i) B1_i, pointers per item via strides
    const int *ia0, *ib0, *ia1, *ib1;   // per item grid indices; results: tmp slots 0, 1 (G space)
    __device__ V xyf_load(int item, int f, int, int, int, size_t p) const
    {
        const size_t N = this->g.N;
        if (f == 0) return cmulc(A0[(size_t)ia0[item] * N + p], B0[(size_t)ib0[item] * N + p]);
        return cmulc(A1[(size_t)ia1[item] * N + p], B1[(size_t)ib1[item] * N + p]);
    }
    __device__ V zmix(int, int o, int, int, int, const V *in) const
    {
        return cscale(in[o], (decltype(in[0].x))this->invN);
    }
    __device__ void xyi_accum(int, int, int, size_t, const V *) const {}
};

// band part of 3a4 / 3b5 (:848-911): targets (k, j), sources (q2sym, i2)
template <typename T>
struct OpBand : OpBase<T> {
    using V = typename C2<T>::t;
    static constexpr const char *NAME = "band";
    static constexpr unsigned BLI = 0xF, BLO = 0xF;
    static constexpr bool ZSPLIT = false;     // one thread per z-line measured faster here
    static constexpr bool REGACC = true;
    __device__ bool regacc_grid(int) const { return true; }
    __device__ V xyi_term(int, int item, int b, size_t p, const V *v) const
    {
        const size_t N = this->g.N;
        const int si = item % this->ns;
        if (b < 3) return cmul(__ldg(&Qt[((size_t)si * 3 + b) * N + p]), v[0]);
        return cscale(cmul(v[0], __ldg(&Rocc[(size_t)si * N + p])), (decltype(v[0].x))(fb5 * fill[si]));
    }
    __device__ void xyi_flush(int tj, size_t p, V s) const { acc_red(acc + (size_t)tj * this->g.N + p, to64(s), 1.0); }
    __device__ const V *xyi_operand(int, int b, int si) const
    {
        return b < 3 ? Qt + ((size_t)si * 3 + b) * this->g.N : Rocc + (size_t)si * this->g.N;
    }
    template <class F> __device__ void xyi_add(int si, int b, const V *v, const V *o, F &&add) const
    {
        const V w = cmul(v[0], o[0]);
        add(0, b < 3 ? w : cscale64(w, fb5 * fill[si]));
    }
    __device__ const V *xyf_operand(int, int f, int si) const
    {
        return f == 0 ? Rchi + (size_t)si * this->g.N : Bt + ((size_t)si * 3 + (f - 1)) * this->g.N;
    }
    __device__ V xyf_pair(int tj, int f, size_t p, const V *o) const
    {
        const V phj = __ldg(&Rpsi[(size_t)tj * this->g.N + p]);
        return f == 0 ? cmulc(o[0], phj) : cmul(o[0], phj);
    }
    static constexpr int ZMO = 3, ZM0 = 1;
    using ZC = typename OpBase<T>::ZC;
    __device__ ZC zctx(int item, int x, int y, int c) const
    {
        ZC z = this->zctx_base(item, x, y, c, 1);
        z.f = (T)(fill[item % this->ns] * fa4);
        return z;
    }
    __device__ T du(const ZC &c, int d, int z) const
    {
        if constexpr (OpBase<T>::FT) return this->zpl(c, d, z);
        else return this->zdu(c, 1, 0, d, z);
    }
    __device__ T zmixc(const ZC &c, int f, int z) const { return du(c, f - 1, z); }
    __device__ T zoutc(const ZC &c, int o, int z) const { return c.f * du(c, o, z); }
    __device__ void xyi_put(int tj, int, int, size_t p, V s) const { xyi_flush(tj, p, s); }
    static constexpr int NF = 4, NB = 4;
    const V *Rpsi;                // [nt][N]
    const V *Rocc, *Rchi;         // phi_q2sym, chi_q2sym [ns][N]
    const V *Qt, *Bt;             // rotated intermediates [ns][3][N]
    double2 *acc;
    const double *fill;           // f2 per source
    double fa4, fb5;
    __device__ V xyf_load(int item, int f, int, int, int, size_t p) const
    {
        const size_t N = this->g.N;
        const int tj = item / this->ns, si = item % this->ns;
        const V phj = __ldg(&Rpsi[(size_t)tj * N + p]);
        if (f == 0) return cmulc(__ldg(&Rchi[(size_t)si * N + p]), phj);   // (:865)
        return cmul(__ldg(&Bt[((size_t)si * 3 + (f - 1)) * N + p]), phj);   // (:885)
    }
    __device__ V zmix(int item, int o, int x, int y, int z, const V *in) const
    {
        using S = decltype(in[0].x);
        if constexpr (OpBase<T>::FT) {
            const size_t p = this->pidx(x, y, z);
            if (o < 3) return cscale(in[0], (float)(fill[item % this->ns] * fa4) * this->fco(item, p, o));
            V r = cscale(in[1], this->fco(item, p, 0));
            r = cadd(r, cscale(in[2], this->fco(item, p, 1)));
            return cadd(r, cscale(in[3], this->fco(item, p, 2)));
        }
        double G[3];
        gvec(this->rc.R, this->g, x, y, z, this->kq_of(item), G);
        const size_t p = this->pidx(x, y, z);
        const double u = this->tab_of(item)[p] * this->invN;
        if (o < 3) {    // f2 a4 phiphi du0_d  (:867-872)
            const double f2 = fill[item % this->ns];
            return cscale(in[0], (S)(f2 * fa4 * G[o] * u));
        }
        V r = cscale(in[1], (S)(G[0] * u));     // sum_d FFT(Bt_d phi_j) du0_d (:882-890)
        r = cadd(r, cscale(in[2], (S)(G[1] * u)));
        return cadd(r, cscale(in[3], (S)(G[2] * u)));
    }
    __device__ void xyi_accum(int tj, int item, int b, size_t p, const V *v) const
    {
        const size_t N = this->g.N;
        const int si = item % this->ns;
        double2 *a = acc + (size_t)tj * N + p;
        if (b < 3) acc_red(a, to64(cmul(__ldg(&Qt[((size_t)si * 3 + b) * N + p]), v[0])), 1.0);    // (:875)
        else acc_red(a, to64(cmul(v[0], __ldg(&Rocc[(size_t)si * N + p]))), fb5 * fill[si]);      // (:894)
    }
};

} // namespace tcg

#include "tc3.cuh"
