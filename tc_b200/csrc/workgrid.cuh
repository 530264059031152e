// workgrid.cuh -- the grid the library works on.
//
// H psi is only needed on the plane-wave sphere of each k (radius at most R =
// max |k+G|), and everything that is multiplied in real space on the way is
// band limited, so a grid coarser than the caller's gives the same sums: a
// product on a grid with periods L folds component G onto G + L, and no folded
// component reaches one that is used as long as the shortest period is longer
// than the sum of the radii of what is computed and what is used.
//   HF: pair densities conj(phi_q) psi_k reach 2 R and are used up to 2 R; the
//   products phi_q X (3 R) and V_H psi (V_H taken up to 2 R: 3 R) are used up to
//   R.  Shortest period > 4 R.
//   TC / BITC: w_d = IFFT[K_d u rho] reaches 2 R, qsum_d = sum f w_d phi_q and the
//   rotated Q, B intermediates 3 R, with density and dnu of 2 R; the products
//   n w_d, conj(chi) qsum_d, B psi (4 R) are used up to 2 R, w_d Q_d and
//   dnu_d qsum_d (5 R) up to R.  Shortest period > 6 R.
// The same must hold for the caller's grid (otherwise its own folded components
// belong to the result), and for TC / BITC the density has to vanish beyond 2 R
// (checked per state: one from orbitals does, a foreign one may not).  When any
// of this fails the caller's grid is used.
//
// For fcc silicon with 14 Ha on 36^3: R = 5.29, |36 b| = 38.2, so HF runs on 20^3
// (|20 b| = 21.21 > 21.17) and TC on 30^3 (31.82 > 31.75).
#pragma once
#include "terms.cuh"

namespace tcg {

// work grid [N] (G space) <- the components of a caller's grid (G space) with
// |G| <= 2 R; the others are zero
static __global__ void k_ball_in(size_t nball, const int2 *map, const double2 *u, double2 *w)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nball; i += (size_t)gridDim.x * blockDim.x)
        w[map[i].y] = u[map[i].x];
}
static __global__ void k_ball_out(size_t nball, const int2 *map, const double2 *w, double2 *u)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < nball; i += (size_t)gridDim.x * blockDim.x)
        u[map[i].x] = w[map[i].y];
}
static int to_work_grid(tcg_ctx *c, const double2 *u, double2 *w)
{
    TCG_CUDA(cudaMemsetAsync(w, 0, (size_t)c->h.N * sizeof(double2), c->stream));
    return launch(c, k_ball_in, dim3(148), dim3(256), 0, c->h.nball, (const int2 *)c->ballmap.as<int2>(), u, w);
}
static int to_user_grid(tcg_ctx *c, const double2 *w, double2 *u)
{
    TCG_CUDA(cudaMemsetAsync(u, 0, (size_t)c->h.uN * sizeof(double2), c->stream));
    return launch(c, k_ball_out, dim3(148), dim3(256), 0, c->h.nball, (const int2 *)c->ballmap.as<int2>(), w, u);
}

// largest |v|^2 of a grid, and of its points outside the sphere |G| <= rad (out[0], out[1]; non-negative
// doubles order like their bits)
static __global__ void __launch_bounds__(256) k_outside(GridDesc g, RecipC rc, double rad2, const double2 *v,
                                                        unsigned long long *out)
{
    double all = 0, off = 0;
    const double zero[3] = {0, 0, 0};
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < g.N; p += gridDim.x * blockDim.x) {
        int x, y, z;
        xyz_of(g, p, x, y, z);
        double G[3];
        gvec(rc.R, g, x, y, z, zero, G);
        const double a = v[p].x * v[p].x + v[p].y * v[p].y;
        all = fmax(all, a);
        if (G[0] * G[0] + G[1] * G[1] + G[2] * G[2] > rad2) off = fmax(off, a);
    }
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        all = fmax(all, __shfl_xor_sync(0xffffffffu, all, o));
        off = fmax(off, __shfl_xor_sync(0xffffffffu, off, o));
    }
    if ((threadIdx.x & 31) == 0) {
        atomicMax(&out[0], (unsigned long long)__double_as_longlong(all));
        atomicMax(&out[1], (unsigned long long)__double_as_longlong(off));
    }
}

static __global__ void k_real_to_complex(int N, const double *a, double2 *b)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) b[p] = {a[p], 0.0};
}
static __global__ void k_real_part(int N, const double2 *a, double *b)
{
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < N; p += gridDim.x * blockDim.x) b[p] = a[p].x;
}
static __global__ void k_drop_imag(size_t n, double2 *a)
{
    for (size_t i = blockIdx.x * (size_t)blockDim.x + threadIdx.x; i < n; i += (size_t)gridDim.x * blockDim.x) a[i].y = 0.0;
}

static inline int signed_miller(int i, int n) { return i <= n / 2 ? i : i - n; }
static inline void miller_of(const Host &h, int gi, int *m)
{
    m[0] = signed_miller(gi % h.un[0], h.un[0]);
    m[1] = signed_miller((gi / h.un[0]) % h.un[1], h.un[1]);
    m[2] = signed_miller(gi / (h.un[0] * h.un[1]), h.un[2]);
}
// grid index of a Miller triple on the work grid
static inline int work_index(const Host &h, const int *m)
{
    int w[3];
    for (int d = 0; d < 3; d++) w[d] = ((m[d] % h.n[d]) + h.n[d]) % h.n[d];
    return w[0] + h.n[0] * (w[1] + h.n[1] * w[2]);
}
// shortest non-zero period of a grid n in reciprocal space
static double shortest_period(const Host &h, const int *n)
{
    double best = 1e300;
    for (int a = -3; a <= 3; a++)
        for (int b = -3; b <= 3; b++)
            for (int c = -3; c <= 3; c++) {
                if (!a && !b && !c) continue;
                const double x[3] = {(double)a * n[0], (double)b * n[1], (double)c * n[2]};
                double v[3];
                cart(h, x, v);
                best = std::min(best, sqrt(v[0] * v[0] + v[1] * v[1] + v[2] * v[2]));
            }
    return best;
}
// |a_i| / (2 pi): Miller extent along axis i of a unit Cartesian length
static double miller_extent(const Host &h, int i)
{
    const double *a = &h.lattice[3 * i];
    return sqrt(a[0] * a[0] + a[1] * a[1] + a[2] * a[2]) / (2.0 * PI_D);
}

// Edge of the cheapest compiled cubic grid that gives the caller's results (0:
// the caller's own).  Sets h.rmax.  That is the smallest, except where its lines
// split badly (15 = 5 x 3, 27 = 9 x 3, 45 = 9 x 5: most threads of the shorter step
// wait) and the next size fits as well or is the caller's own.  An apply at the
// cutoff of the smaller size, ms on it and on the next:
//            FP32 TC      HF            FP64 TC      HF
//   15, 16   0.96  0.88   0.129 0.120   1.47  1.45   0.173 0.164   next in both
//   27, 30   5.15  5.20   0.81  0.85    12.5  9.12   1.41  1.32    next in FP64
//   45, 48   0.88  0.91   0.217 0.214   1.51  1.46   0.290 0.293   next in FP64 TC
static int choose_reduced(Host &h, bool fp64)
{
    h.rmax = 0;
    int mmax[3] = {0, 0, 0};
    for (int s = 0; s < h.nspin; s++)
        for (int a = 0; a < h.nk_all; a++) {
            double q[3];
            cart(h, &h.kvec[3 * a], q);
            const size_t o = h.gidx_off[(size_t)s * h.nk_all + a];
            for (int p = 0; p < h.npw[h.ik_of_all[a]]; p++) {
                int m[3];
                miller_of(h, h.gidx_host[o + p], m);
                const double x[3] = {(double)m[0], (double)m[1], (double)m[2]};
                double G[3];
                cart(h, x, G);
                double r = 0;
                for (int d = 0; d < 3; d++) {
                    r += (G[d] + q[d]) * (G[d] + q[d]);
                    mmax[d] = std::max(mmax[d], std::abs(m[d]));
                }
                h.rmax = std::max(h.rmax, sqrt(r));
            }
        }
    const bool hf = h.method == TCG_METHOD_HF;
    const double need = (hf ? 4.0 : 6.0) * h.rmax * (1.0 + 1e-6);
    if (!(shortest_period(h, h.un) > need)) return 0;
    auto integral = [&](int n, int d) {        // fractional translations on the grid (rotation phases)
        for (int o = 0; o < h.nsymop; o++) {
            const double x = h.translation[3 * o + d] * n;
            if (fabs(x - nearbyint(x)) > 1e-9) return false;
        }
        return true;
    };
    const bool user_fast = h.un[0] == h.un[1] && h.un[1] == h.un[2] && fast_grid(h.un[0]);
    if (!hf)
        for (int d = 0; d < 3; d++)
            if (!integral(h.un[d], d)) return 0;
    int best = 0;
    bool done = false;                         // the size after the smallest has been looked at
    auto consider = [&](int n) {
        const int n3[3] = {n, n, n};
        const double pts = (double)n * n * n;
        if (best) {
            if (done) return;
            done = true;
            if (!(best == 15 || (fp64 && (best == 27 || (best == 45 && !hf))))) return;
            if (h.un[0] == n && h.un[1] == n && h.un[2] == n) {
                best = 0;
                return;
            }
        }
        if (pts > (user_fast ? 0.9 : 1.0) * h.uN) return;
        if (!(shortest_period(h, n3) > need)) return;
        for (int d = 0; d < 3; d++) {
            if (2 * mmax[d] >= n) return;      // the plane waves keep their signed indices
            if (hf) continue;
            if (!integral(n, d)) return;
            // so do the pair densities: centre k - q, radius 2 R
            for (int k = 0; k < h.nk; k++)
                for (int a = 0; a < h.nk_all; a++) {
                    const double ci = h.kvec[3 * h.kall_off[k] + d] - h.kvec[3 * a + d];
                    const double reach = fabs(ci) + 2.0 * h.rmax * (1.0 + 1e-9) * miller_extent(h, d);
                    if (reach >= (n - 1) / 2.0 || reach >= (h.un[d] - 1) / 2.0) return;
                }
        }
        best = n;
    };
#define TCG_TRY(m) consider(m);
    TCG_FAST_SIZES(TCG_TRY)
#undef TCG_TRY
    return best;
}

// FP32 twiddle: of the floats next to each component, the pair with the modulus
// closest to 1, the direction weighing less.  Nearest rounding shortens or
// lengthens the factors of some lengths on average (16: -1.1e-8 per line
// transform, -2e-10 so), which adds up along a chain of transforms.
static float2 round_twiddle(double re, double im)
{
    auto near0 = [](double x) { return fabs(x) < 1e-9; };
    const float r0 = near0(re) ? 0.f : (float)re, i0 = near0(im) ? 0.f : (float)im;
    float2 best = make_float2(r0, i0);
    double cost = 1e300;
    for (int a = -1; a <= 1; a++)
        for (int b = -1; b <= 1; b++) {
            if ((a && r0 == 0.f) || (b && i0 == 0.f)) continue;
            const float r = a ? nextafterf(r0, a * 9.f) : r0, i = b ? nextafterf(i0, b * 9.f) : i0;
            const double m = sqrt((double)r * r + (double)i * i) - 1.0, ex = r - re, ey = i - im;
            const double c = m * m + 0.0225 * (ex * ex + ey * ey);
            if (c < cost) {
                cost = c;
                best = make_float2(r, i);
            }
        }
    return best;
}

// device twiddles and description of a grid
static int make_grid(tcg_ctx *c, const int *n, GridDesc &g, DBuf &tw64, DBuf &tw32)
{
    g.n0 = n[0]; g.n1 = n[1]; g.n2 = n[2]; g.N = n[0] * n[1] * n[2];
    for (int d = 0; d < 3; d++) TRY(make_axis(n[d], g.ax[d]));
    std::vector<double2> t64(3 * MAXN);
    std::vector<float2> t32(3 * MAXN);
    for (int d = 0; d < 3; d++)
        for (int j = 0; j < n[d]; j++) {
            const long double a = 2.0L * (long double)PI_D * j / n[d];
            const double cr = (double)cosl(a), ci = -(double)sinl(a);
            t64[d * MAXN + j] = make_double2(cr, ci);
            t32[d * MAXN + j] = round_twiddle(cr, ci);
        }
    TRY(up(tw64, t64.data(), t64.size() * sizeof(double2), c->stream));
    TRY(up(tw32, t32.data(), t32.size() * sizeof(float2), c->stream));
    TCG_CUDA(cudaStreamSynchronize(c->stream));
    g.tw64 = tw64.as<const double2>();
    g.tw32 = tw32.as<const float2>();
    if (&g == &c->gd) {
        c->htw64.assign(t64.begin(), t64.begin() + n[0]);
        c->htw32.assign(t32.begin(), t32.begin() + n[0]);
    }
    return TCG_OK;
}

static int build_prune_table(tcg_ctx *c);

// the local pseudopotential uvloc on the work grid (u, w: scratch on the two grids)
static int place_vloc_on(tcg_ctx *c, double2 *u, double2 *w)
{
    const Host &h = c->h;
    TRY(launch(c, k_real_to_complex, dim3(148), dim3(256), 0, h.uN, (const double *)c->uvloc.p, u));
    std::vector<void *> gu{u}, gw{w};
    TRY((fft3_list<double, -1>(c, gu, &c->ugd)));
    TRY(to_work_grid(c, u, w));
    TRY((fft3_list<double, +1>(c, gw)));
    return launch(c, k_real_part, dim3(148), dim3(256), 0, h.N, (const double2 *)w, c->vloc.as<double>());
}
static int place_vloc(tcg_ctx *c)
{
    const Host &h = c->h;
    TRY(c->vloc.ensure((size_t)h.N * sizeof(double)));
    if (!h.reduced) {
        TCG_CUDA(cudaMemcpyAsync(c->vloc.p, c->uvloc.p, (size_t)h.N * sizeof(double), cudaMemcpyDeviceToDevice, c->stream));
        return TCG_OK;
    }
    DBuf work;
    TRY(work.ensure((size_t)(h.uN + h.N) * sizeof(double2)));
    double2 *u = work.as<double2>(), *w = u + h.uN;
    const int rc = place_vloc_on(c, u, w);
    cudaStreamSynchronize(c->stream);
    work.release();
    return rc;
}

// Set up the work grid: the caller's, or red_n^3.  When it fails half-way, c->grid_ok
// stays clear and the next user of the grid sets it up again.
static int configure_grid(tcg_ctx *c, bool reduced)
{
    Host &h = c->h;
    c->grid_ok = false;
    TCG_CUDA(cudaStreamSynchronize(c->stream));
    h.reduced = reduced;
    for (int d = 0; d < 3; d++) h.n[d] = reduced ? h.red_n : h.un[d];
    h.N = h.n[0] * h.n[1] * h.n[2];
    TRY(make_grid(c, h.n, c->gd, c->tw64, c->tw32));
    c->fast_n = h.n[0] == h.n[1] && h.n[1] == h.n[2] && fast_grid(h.n[0]) ? h.n[0] : 0;
    // grid point -> plane wave of every (spin, all-k), plane wave -> grid point at isym 0
    std::vector<int> inv((size_t)h.nspin * h.nk_all * h.N, -1), g0;
    h.g0_off.resize((size_t)h.nspin * h.nk);
    for (int s = 0; s < h.nspin; s++)
        for (int a = 0; a < h.nk_all; a++) {
            const int k = h.ik_of_all[a];
            const size_t o = h.gidx_off[(size_t)s * h.nk_all + a];
            int *im = inv.data() + ((size_t)s * h.nk_all + a) * h.N;
            if (a == h.kall_off[k]) h.g0_off[(size_t)s * h.nk + k] = g0.size();
            for (int p = 0; p < h.npw[k]; p++) {
                int gi = h.gidx_host[o + p];
                if (reduced) {
                    int m[3];
                    miller_of(h, gi, m);
                    gi = work_index(h, m);
                }
                im[gi] = p;
                if (a == h.kall_off[k]) g0.push_back(gi);
            }
        }
    TRY(up(c->inv, inv.data(), inv.size() * sizeof(int), c->stream));
    TRY(up(c->gidx0, g0.data(), g0.size() * sizeof(int), c->stream));
    TCG_CUDA(cudaStreamSynchronize(c->stream));
    h.hf_wrap = false;
    if (reduced) {
        std::vector<int2> map;
        const double r2 = 4.0 * h.rmax * h.rmax * (1.0 + 1e-9);
        int e[3];
        for (int d = 0; d < 3; d++) e[d] = (int)ceil(2.0 * h.rmax * miller_extent(h, d)) + 1;
        for (int z = -e[2]; z <= e[2]; z++)
            for (int y = -e[1]; y <= e[1]; y++)
                for (int x = -e[0]; x <= e[0]; x++) {
                    const int m[3] = {x, y, z};
                    const double xm[3] = {(double)x, (double)y, (double)z};
                    double G[3];
                    cart(h, xm, G);
                    if (G[0] * G[0] + G[1] * G[1] + G[2] * G[2] > r2) continue;
                    int u[3];
                    for (int d = 0; d < 3; d++) u[d] = ((m[d] % h.un[d]) + h.un[d]) % h.un[d];
                    map.push_back(make_int2(u[0] + h.un[0] * (u[1] + h.un[1] * u[2]), work_index(h, m)));
                }
        h.nball = map.size();
        TRY(up(c->ballmap, map.data(), map.size() * sizeof(int2), c->stream));
        TCG_CUDA(cudaStreamSynchronize(c->stream));
        h.hf_wrap = h.method == TCG_METHOD_HF;
    }
    c->hftab_ok = false;
    c->prune_ok = false;
    c->any_ok = !c->fast_n && sl::any_shape(h.n, c->prec == TCG_PREC_FP64 ? sizeof(double2) : sizeof(float2), c->any);
    if (c->fast_n || c->any_ok) TRY(build_prune_table(c));
    if (h.have_vloc) TRY(place_vloc(c));
    c->grid_ok = true;
    return TCG_OK;
}
// The kernel forms in use run on the smaller grid: split lines, by default or by number
static bool forms_reduce(const tcg_ctx *c)
{
    return c->h.red_n && (c->xy_kernels == 0 || c->xy_kernels == 3) && (c->z_kernels == 0 || c->z_kernels >= 3) && !c->force_generic;
}
static int ensure_grid(tcg_ctx *c) { return c->grid_ok ? TCG_OK : configure_grid(c, c->h.reduced); }

// Choose the work grid for the state whose density is in c->udens and bring the
// density onto it.
static int place_state(tcg_ctx *c)
{
    Host &h = c->h;
    const bool hf = h.method == TCG_METHOD_HF;
    const size_t uN = h.uN;
    bool want = forms_reduce(c);
    if (want && !hf) {
        // density in G; its largest component beyond 2 R against its largest
        TRY(c->uwork.ensure(2 * uN * sizeof(double2) + 4 * sizeof(unsigned long long)));
        double2 *u = c->uwork.as<double2>();
        unsigned long long *mx = reinterpret_cast<unsigned long long *>(u + 2 * uN);
        TCG_CUDA(cudaMemcpyAsync(u, c->udens.p, 2 * uN * sizeof(double2), cudaMemcpyDeviceToDevice, c->stream));
        TCG_CUDA(cudaMemsetAsync(mx, 0, 4 * sizeof(unsigned long long), c->stream));
        std::vector<void *> gu{u, u + uN};
        TRY((fft3_list<double, -1>(c, gu, &c->ugd)));
        RecipC rc;
        memcpy(rc.R, h.recip, sizeof rc.R);
        const double r2 = 4.0 * h.rmax * h.rmax * (1.0 + 1e-9);
        for (int s = 0; s < 2; s++)
            TRY(launch(c, k_outside, dim3(148), dim3(256), 0, c->ugd, rc, r2, (const double2 *)(u + s * uN), mx + 2 * s));
        double m2[4];
        TCG_CUDA(cudaMemcpyAsync(m2, mx, sizeof m2, cudaMemcpyDeviceToHost, c->stream));
        TCG_CUDA(cudaStreamSynchronize(c->stream));
        // 1e-13 in amplitude: rounding of the transforms that made it is some 1e-16
        for (int s = 0; s < 2; s++)
            if (!(m2[2 * s + 1] <= 1e-26 * m2[2 * s])) want = false;
    }
    if (want != h.reduced || !c->grid_ok) TRY(configure_grid(c, want));
    if (hf) return TCG_OK;
    TRY(c->dens.ensure(2 * (size_t)h.N * sizeof(double2)));
    if (!h.reduced) {
        TCG_CUDA(cudaMemcpyAsync(c->dens.p, c->udens.p, 2 * uN * sizeof(double2), cudaMemcpyDeviceToDevice, c->stream));
        return TCG_OK;
    }
    for (int s = 0; s < 2; s++) {
        double2 *w = c->dens.as<double2>() + (size_t)s * h.N;
        TRY(to_work_grid(c, c->uwork.as<double2>() + s * uN, w));
    }
    std::vector<void *> gw{c->dens.as<double2>(), c->dens.as<double2>() + h.N};
    return fft3_list<double, +1>(c, gw);
}

} // namespace tcg
