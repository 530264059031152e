// ctx.cuh -- the library context: device copies of the system / state,
// FFT plans, scratch arenas, launch helpers.
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>
#include <string>
#include <vector>
#include <unordered_set>
#include "../../include/tcg.h"
#include "fft.cuh"

namespace tcg {

void set_error(const char *fmt, ...);

struct Status {
    int code = TCG_OK;
};

#define TCG_CUDA(call)                                                                    \
    do {                                                                                  \
        cudaError_t e_ = (call);                                                          \
        if (e_ != cudaSuccess) {                                                          \
            tcg::set_error("CUDA error %s at %s:%d (%s)", cudaGetErrorString(e_), __FILE__, \
                           __LINE__, #call);                                              \
            return TCG_ERR_CUDA;                                                          \
        }                                                                                 \
    } while (0)

// Failure injection of tests (tcg_debug_fail_alloc): the n-th allocation of a DBuf by
// this thread fails; 0: none does.
inline thread_local int g_fail_alloc = 0;

// Device buffer (owned).
struct DBuf {
    void *p = nullptr;
    size_t bytes = 0;
    int ensure(size_t b)
    {
        if (b <= bytes) return TCG_OK;
        // kernels queued earlier may still read the old buffer
        if (p) { cudaDeviceSynchronize(); cudaFree(p); }
        p = nullptr;
        bytes = 0;
        if (b == 0) return TCG_OK;
        if ((g_fail_alloc > 0 && --g_fail_alloc == 0) || cudaMalloc(&p, b) != cudaSuccess) {
            cudaGetLastError();
            p = nullptr;
            set_error("cudaMalloc of %zu bytes failed", b);
            return TCG_ERR_NOMEM;
        }
        bytes = b;
        return TCG_OK;
    }
    void release()
    {
        if (p) cudaFree(p);
        p = nullptr;
        bytes = 0;
    }
    template <typename X> X *as() const { return reinterpret_cast<X *>(p); }
};

struct Host {
    // system
    int un[3] = {0, 0, 0}, uN = 0;          // the caller's FFT grid
    int n[3] = {0, 0, 0}, N = 0;            // the grid the library works on (workgrid.cuh)
    int red_n = 0;                          // edge of the smaller work grid this geometry allows (0: none)
    bool reduced = false;                   // the work grid is red_n^3 instead of the caller's
    bool hf_wrap = false;                   // pair-density spheres may wrap around the work grid's box (HF)
    double rmax = 0;                        // largest |k+G| of any plane wave
    size_t nball = 0;                       // entries of ballmap
    double recip[9], lattice[9], omega = 0;
    int method = 0, nspin = 1, nk = 0, nk_all = 0, num_kpoints = 0;
    std::vector<int> nsym_k, kall_off, ik_of_all, npw;
    std::vector<double> kvec;               // [nk_all][3]
    std::vector<uint8_t> time_rev;
    std::vector<int> rot_index;
    int nsymop = 0;
    std::vector<int> rotation;              // [nsymop][9]
    std::vector<double> translation;        // [nsymop][3]
    std::vector<size_t> gidx_off;           // [nspin*nk_all] offset in gindex / phase
    std::vector<int> gidx_host;             // host copy of gindex (on the caller's grid)
    double A[4], F[4];
    bool A_zero = true;
    bool div = false;
    double alpha = 0;
    std::vector<double> sum_vaux;
    // state
    bool have_state = false;
    std::vector<int> nbands, nocc;          // [nspin], [nspin][nk]
    std::vector<double> filling;            // [nspin][nk][nbands]
    std::vector<size_t> orb_off;            // [nspin*nk] complex offset of band 0
    std::vector<size_t> occ_off;            // [nspin*nk_all] grid offset into Rocc
    size_t nocc_grids = 0;
    bool qp_ready = false;                  // tc3a2a4b2b5 occupied-pair stage done for this state
    bool qp_pending = false;                // a partial stage awaits the caller's sum and tcg_qp_finish
    // one-body data
    bool have_pseudo = false, have_vloc = false;
    int nl_ncomp = 0;                       // projector components (atom, projector, m)
    std::vector<size_t> nl_koff;            // [nk] offset of k in nlB
    size_t nl_dval_off = 0;                 // byte offset of the D values in nlD
    std::vector<size_t> g0_off;             // [nspin*nk] offset of (s, k) in gidx0
};

// cubic grid sizes with compiled pass kernels: split lines (split.cuh) at all of
// them, one thread or a lane pair per line (fast.cuh) at line_grid's
#define TCG_FAST_SIZES(X) X(12) X(15) X(16) X(18) X(20) X(24) X(25) X(27) X(30) X(32) X(36) X(40) X(45) X(48)
inline bool fast_grid(int n)
{
#define TCG_IS(m) if (n == m) return true;
    TCG_FAST_SIZES(TCG_IS)
#undef TCG_IS
    return false;
}
constexpr bool line_grid(int n) { return n == 12 || n == 16 || n == 24 || n == 32 || n == 36 || n == 40 || n == 48; }
// grids on which tcg_set_forms offers the split-line forms by number
inline bool split_line_grid(int n) { return n == 36 || n == 48; }

namespace sl {
// run-time shape of the split-line passes on other grids (anygrid.cuh): n = a b
// along each axis, row stride and size of an XY buffer
struct AnyShape {
    int n[3], a[3], b[3], rs, ps;
};
constexpr int MAXTHR = 9 * 64;       // threads of an XY pass: a (<= 9) per line, 64 lines

inline bool any_shape(const int *n, size_t vbytes, AnyShape &s)
{
    for (int d = 0; d < 3; d++) {
        s.n[d] = n[d];
        s.a[d] = 0;
        for (int a = 9; a >= 2; a--)
            if (n[d] <= 64 && n[d] % a == 0 && n[d] / a <= a && n[d] / a >= 2) { s.a[d] = a; s.b[d] = n[d] / a; }
        if (!s.a[d]) return false;
    }
    const int m = n[0] > n[1] ? n[0] : n[1];
    s.rs = m | 1;
    s.ps = s.rs * m;
    const int thr = s.a[1] * n[0] > s.a[0] * n[1] ? s.a[1] * n[0] : s.a[0] * n[1];
    // the inverse XY pass with three sums per point, the Z pass with six inputs
    return vbytes * (n[0] + n[1] + 2 * (size_t)s.ps + 3 * (size_t)s.b[1] * thr) <= 227 * 1024 &&
           vbytes * (size_t)n[2] * (1 + 6 * 32) <= 227 * 1024;
}
} // namespace sl

// layout of the pencil table of pruned transforms: bits [nent][n1] u64,
// counts [nent] int, permutations [nent][n0 n1] u16
struct PruneTable {
    size_t nent, np, nact, perm, bytes;
    explicit PruneTable(const Host &h)
        : nent((size_t)h.nk * h.nk_all), np((size_t)h.n[0] * h.n[1]), nact(nent * h.n[1] * 8), perm(nact + nent * 4),
          bytes(perm + nent * np * 2) {}
};

struct tcg_ctx_impl;
} // namespace tcg

struct tcg_ctx {
    int device = 0;
    int prec = TCG_PREC_FP64;
    cudaStream_t stream = nullptr;
    tcg::Host h;
    tcg::GridDesc gd;
    // static device data
    tcg::GridDesc ugd;                      // the caller's grid (gd: the work grid)
    tcg::DBuf utw64, utw32;
    tcg::DBuf ballmap;                      // [nball] int2: caller's grid index, work grid index (workgrid.cuh)
    tcg::DBuf udens, uvloc, uwork;          // density / local pseudopotential / scratch on the caller's grid
    tcg::DBuf tw64, tw32, recip;            // twiddles, reciprocal vectors (9 doubles)
    tcg::DBuf inv;                          // [nspin][nk_all][N] int32
    tcg::DBuf phase;                        // [sum npw] double2
    // state
    tcg::DBuf phik, chik;                   // G-space fp64 (chik only for BITC)
    tcg::DBuf fill;                         // [nspin][nk][nbands] doubles
    tcg::DBuf Rocc, Rchi, Rgrad;            // R-space occupied grids (compute precision)
    tcg::DBuf dens;                         // [2][N] double2
    tcg::DBuf densT;                        // [3][N] compute precision: n_0, n_1, n_0 + n_1
    tcg::DBuf occfill;                      // [nocc_grids] doubles: filling of each occupied grid
    // local three-body potentials built per state
    tcg::DBuf Vloc;                         // [nspin][N] double2 (tc3a1 + tc3b1 + ...)
    tcg::DBuf dnu, dnuT;                    // [nspin][3][N] fp64 / compute precision
    tcg::DBuf V3a1, V3b1, V3a2, V3b2;       // [nspin][N] fp64 local three-body potentials
    tcg::DBuf VH;                           // [N] fp64 Hartree potential (hf2h)
    tcg::DBuf V2h;                          // [nspin][N] fp64 TC Hartree potential (tc2h [2a_h] + [2b_h2])
    tcg::DBuf pgw;                          // [3][N] fp64 work: sum_q f conj(chi_q) grad phi_q (tc2h [2b_h2])
    // one-body data (tcg_set_pseudo) and per-apply scratch
    tcg::DBuf gidx0;                        // [nspin][sum npw] grid index of each plane wave at isym 0
    tcg::DBuf vloc;                         // [N] fp64 local pseudopotential (real), or empty
    tcg::DBuf nlB;                          // [sum_k ncomp npw_k] complex exp(iG.R) x projector
    tcg::DBuf nlD;                          // CSR of D between projector components
    tcg::DBuf acc1, h1buf;                  // one-body accumulators / device copies
    tcg::DBuf gpsi, adjw, adjt;             // energy gradients: occupied block + outputs, pair grids, tables
    // pruned transforms: per (irreducible k, all-k q) pair, the
    // (x, y) pencils of the grid that the support of a pair density touches
    tcg::DBuf prune_tab;                    // PruneTable
    bool prune_ok = false;                  // table built and usable
    std::vector<int> prune_nact;            // host copy of the table's active-pencil counts
    bool no_prune = false;                  // TCG_NO_PRUNE: full transforms everywhere
    bool use_sacc = false;                  // tcg_forms.sacc / .qp_sacc: kept as set, no kernel asks for them
    bool qp_sacc = true;
    bool no_fuse = false;                   // TCG_NO_FUSE: tc2x and tc3a3b3b4b6 run as separate passes
    tcg::DBuf Qt, Bt;                       // tc3a2a4b2b5 rotated intermediates [nocc_grids][3][N]
    tcg::DBuf accP, qtg;                    // occupied-pair accumulators / gathered q2 grids
    tcg::DBuf div3b6;                       // [nspin][N] fp64 temp_div_3b6 in R space
    std::vector<double2> t1_3b6;            // [nspin][nk] temp_div_3b6_1
    // per-apply scratch
    tcg::DBuf psi, h2, h3;                  // packed fp64
    tcg::DBuf Rpsi, Rgpsi, acc2, acc3, qsum, tmp, tmp2, aux, items, meta;
    tcg::DBuf rotw, q3b2w, nGw, Ww;           // per-state scratch kept across states (no per-step cudaMalloc / cudaFree)
    tcg::DBuf ftab;                         // mixed path: FP32 G-space coefficient planes of a chunk
    tcg::DBuf w3x;                          // [targets][3][N] compute precision: b3 dnu_d psi + b4 qsum_d (3bX input)
    int ftab_nrec = 1;
    tcg::DBuf hftab;                        // hf2x on chip (cube.cuh): kernel of every (irreducible k, all-k q) pair
    bool hftab_ok = false;                  // built for the current work grid
    std::vector<double2> htw64;             // host copies of the work grid's axis-0 twiddles
    std::vector<float2> htw32;
    int fast_n = 0;                         // cubic grid size with compiled fast kernels (0: generic path)
    bool any_ok = false;                    // split-line passes with the run-time shape `any` (fast_n == 0)
    tcg::sl::AnyShape any;
    bool force_generic = false;             // use the generic pass kernels even if fast_n is set
    int xy_kernels = 0;                     // fast XY passes: 0 default (split lines), 1 all line, 2 all lane-pair, 3 split lines
    bool no_prefetch = false;               // fast XYI: no prefetch of the next plane set
    const char *stage = "misc";            // profiling tag of untagged launches (the current stage)
    int z_kernels = 0;                      // fast Z pass: 0 default (split lines), 1 one thread per line, 2 lane
                                            // pairs, 3 and 4 split lines
    size_t tmp_budget = 0;                  // bytes per chunk of pass temporaries (0: default 8 GiB)
    int min_targets = 0;                    // targets per chunk (0: default, about 12 waves of XYI CTAs)
    int64_t launches = 0;
    // optional per-kernel timing with CUDA events on the context stream
    bool prof = false;
    struct ProfRec { const void *fn; const char *tag; cudaEvent_t a, b; double bytes; };
    std::vector<ProfRec> prof_recs;
    bool grid_ok = false;                   // the work grid's tables are complete (configure_grid)
};

namespace tcg {
// split-line XY / Z passes in use (the defaults where compiled); sizes without
// the other forms use them for both or not at all
inline bool split_form(const tcg_ctx *c, bool xy)
{
    const bool fx = c->xy_kernels == 0 || c->xy_kernels == 3, fz = c->z_kernels == 0 || c->z_kernels >= 3;
    if (c->force_generic) return false;
    if (!c->fast_n) return c->any_ok && fx && fz;
    return line_grid(c->fast_n) ? (xy ? fx : fz) : (fx && fz);
}
inline bool split_xy(const tcg_ctx *c) { return split_form(c, true); }
inline bool split_z(const tcg_ctx *c) { return split_form(c, false); }
} // namespace tcg
