// subspace.cu -- the dense band-by-band part of the block Davidson on the
// device, in FP64 (Diagonalization::block_davidson, diagonalization_davidson.cpp:
// 462-600; diagonalization_utils.cpp:7-119):
//   tcg_subspace_ritz   H_n,sub = Vref^H (H_n V) (ZGEMM), H_sub = sum_n H_n,sub,
//                       H_sub X = X D (general complex eigensolve, in one CTA
//                       up to order EIG_MAX, cuSOLVER Xgeev beyond), eigenpairs
//                       sorted by the real part, X^-1 (LU), Ritz vectors V X and
//                       left vectors Vref (X^-1)^H (ZGEMM),
//                       energies diag(Xl^H H_n,sub X)
//   tcg_gram_schmidt    Gram_Schmidt / Gram_Schmidt_biortho of a block of vectors
//   tcg_davidson_expand the new trial vectors of one block: preconditioned
//                       residuals (make_a_new_trial_vector), each orthonormalised
//                       against the basis and appended unless it vanishes
// The band-by-band contractions are plain library GEMMs (cuBLAS ZGEMM runs
// them on the FP64 tensor pipe); the LU is cuSOLVER's.
#include <algorithm>
#include <cmath>
#include <cstring>
#include <mutex>
#include <numeric>
#include <vector>

#include <cublas_v2.h>
#include <cuda_runtime.h>
#include <cusolverDn.h>

#include "../../include/tcg.h"

namespace tcg {
void set_error(const char *fmt, ...);
}

namespace {

int fail(int code, const char *msg)
{
    tcg::set_error("%s", msg);
    return code;
}

#define SUB_CUDA(call)                                                                                        \
    do {                                                                                                      \
        cudaError_t e_ = (call);                                                                              \
        if (e_ != cudaSuccess) {                                                                              \
            tcg::set_error("CUDA error %s at %s:%d", cudaGetErrorString(e_), __FILE__, __LINE__);             \
            return TCG_ERR_CUDA;                                                                              \
        }                                                                                                     \
    } while (0)
#define SUB_BLAS(call)                                                                                        \
    do {                                                                                                      \
        cublasStatus_t e_ = (call);                                                                           \
        if (e_ != CUBLAS_STATUS_SUCCESS) {                                                                    \
            tcg::set_error("cuBLAS error %d at %s:%d", (int)e_, __FILE__, __LINE__);                          \
            return TCG_ERR_CUDA;                                                                              \
        }                                                                                                     \
    } while (0)
#define SUB_SOLV(call)                                                                                        \
    do {                                                                                                      \
        cusolverStatus_t e_ = (call);                                                                         \
        if (e_ != CUSOLVER_STATUS_SUCCESS) {                                                                  \
            tcg::set_error("cuSOLVER error %d at %s:%d", (int)e_, __FILE__, __LINE__);                        \
            return TCG_ERR_CUDA;                                                                              \
        }                                                                                                     \
    } while (0)

struct Handles {
    cublasHandle_t blas = nullptr;
    cusolverDnHandle_t solver = nullptr;
    cusolverDnParams_t params = nullptr;
};
std::mutex g_mu;
Handles g_h[64];
cudaMemPool_t g_pool[64];

// Scratch of the calls comes from a stream-ordered pool per device (safe for
// several threads and streams) that keeps at most 64 MB between calls; cudaMalloc
// and cudaFree took 2 of the 2.5 ms of an expansion.
int scratch_pool(cudaMemPool_t *out)
{
    int dev = 0;
    SUB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(TCG_ERR_UNSUPPORTED, "device index >= 64");
    std::lock_guard<std::mutex> lk(g_mu);
    if (!g_pool[dev]) {
        cudaMemPoolProps props = {};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool;
        SUB_CUDA(cudaMemPoolCreate(&pool, &props));
        unsigned long long keep = 64ull << 20;
        SUB_CUDA(cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep));
        g_pool[dev] = pool;
    }
    *out = g_pool[dev];
    return TCG_OK;
}

int handles(Handles **out)
{
    int dev = 0;
    SUB_CUDA(cudaGetDevice(&dev));
    if (dev < 0 || dev >= 64) return fail(TCG_ERR_UNSUPPORTED, "device index >= 64");
    std::lock_guard<std::mutex> lk(g_mu);
    Handles &h = g_h[dev];
    if (!h.blas) {
        SUB_BLAS(cublasCreate(&h.blas));
        SUB_SOLV(cusolverDnCreate(&h.solver));
        SUB_SOLV(cusolverDnCreateParams(&h.params));
    }
    *out = &h;
    return TCG_OK;
}

// scratch of one call: one allocation on the call's stream, parts handed out in order, freed on return
struct Scratch {
    char *base = nullptr;
    size_t used = 0, cap = 0;
    cudaStream_t st;
    explicit Scratch(cudaStream_t s) : st(s) {}
    ~Scratch()
    {
        if (base) cudaFreeAsync(base, st);
    }
    static size_t part(size_t bytes) { return (std::max<size_t>(bytes, 16) + 255) / 256 * 256; }
    int reserve(size_t bytes)
    {
        cudaMemPool_t pool;
        const int rc = scratch_pool(&pool);
        if (rc) return rc;
        cap = std::max<size_t>(bytes, 256);
        if (cudaMallocFromPoolAsync((void **)&base, cap, pool, st) != cudaSuccess) {
            cudaGetLastError();
            base = nullptr;
            return fail(TCG_ERR_NOMEM, "device allocation failed");
        }
        return TCG_OK;
    }
    template <typename X> X *get(size_t n)
    {
        X *p = reinterpret_cast<X *>(base + used);
        used += part(n * sizeof(X));
        return p;
    }
};

__global__ void k_add3(int n, const double2 *a, const double2 *b, const double2 *c, double2 *out)
{
    const int i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double2 s = {0, 0};
    if (a) s = {s.x + a[i].x, s.y + a[i].y};
    if (b) s = {s.x + b[i].x, s.y + b[i].y};
    if (c) s = {s.x + c[i].x, s.y + c[i].y};
    out[i] = s;
}

// column permutation (col-major n x n): out[:, j] = in[:, perm[j]]
__global__ void k_permute_cols(int n, const int *perm, const double2 *in, double2 *out)
{
    const int j = blockIdx.x;
    for (int r = threadIdx.x; r < n; r += blockDim.x) out[(size_t)j * n + r] = in[(size_t)perm[j] * n + r];
}

// identity (col-major n x n)
__global__ void k_identity(int n, double2 *a)
{
    const int j = blockIdx.x;
    for (int r = threadIdx.x; r < n; r += blockDim.x) a[(size_t)j * n + r] = make_double2(r == j ? 1.0 : 0.0, 0.0);
}

// conjugate transpose (col-major n x n)
__global__ void k_adjoint(int n, const double2 *in, double2 *out)
{
    const int j = blockIdx.x;
    for (int r = threadIdx.x; r < n; r += blockDim.x) {
        const double2 v = in[(size_t)r * n + j];
        out[(size_t)j * n + r] = make_double2(v.x, -v.y);
    }
}

// e[i] = sum_{a,b} conj(L[a,i]) H[a,b] X[b,i]   (col-major, i < nout)
__global__ void k_diag_form(int n, int nout, const double2 *L, const double2 *H, const double2 *X, double2 *e)
{
    const int i = blockIdx.x;
    if (i >= nout) return;
    __shared__ double2 red[256];
    double2 s = {0, 0};
    for (int ab = threadIdx.x; ab < n * n; ab += blockDim.x) {
        const int a = ab % n, b = ab / n;
        const double2 l = L[(size_t)i * n + a], h = H[(size_t)b * n + a], x = X[(size_t)i * n + b];
        const double2 hx = {h.x * x.x - h.y * x.y, h.x * x.y + h.y * x.x};
        s.x += l.x * hx.x + l.y * hx.y;
        s.y += l.x * hx.y - l.y * hx.x;
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] = {red[threadIdx.x].x + red[threadIdx.x + k].x,
                                                 red[threadIdx.x].y + red[threadIdx.x + k].y};
        __syncthreads();
    }
    if (threadIdx.x == 0) e[i] = red[0];
}

// one step of Gram-Schmidt on vector j: target -= <ref_i|target> basis_i for
// i < j, in order (modified Gram-Schmidt, as the reference's loop updates the
// target after each projection); one block
__global__ void k_gs_project(int npw, int j, const double2 *ref, const double2 *basis, double2 *target)
{
    __shared__ double2 red[256];
    for (int i = 0; i < j; i++) {
        const double2 *r = ref + (size_t)i * npw;
        double2 s = {0, 0};
        for (int p = threadIdx.x; p < npw; p += blockDim.x) {
            const double2 a = r[p], b = target[p];
            s.x += a.x * b.x + a.y * b.y;
            s.y += a.x * b.y - a.y * b.x;
        }
        red[threadIdx.x] = s;
        __syncthreads();
        for (int k = blockDim.x / 2; k > 0; k >>= 1) {
            if (threadIdx.x < k) red[threadIdx.x] = {red[threadIdx.x].x + red[threadIdx.x + k].x,
                                                     red[threadIdx.x].y + red[threadIdx.x + k].y};
            __syncthreads();
        }
        const double2 c = red[0];
        __syncthreads();
        const double2 *bs = basis + (size_t)i * npw;
        for (int p = threadIdx.x; p < npw; p += blockDim.x) {
            const double2 b = bs[p];
            target[p].x -= c.x * b.x - c.y * b.y;
            target[p].y -= c.x * b.y + c.y * b.x;
        }
        __syncthreads();
    }
}

// <a|b> into out (one block)
__global__ void k_dotc(int npw, const double2 *a, const double2 *b, double2 *out)
{
    __shared__ double2 red[256];
    double2 s = {0, 0};
    for (int p = threadIdx.x; p < npw; p += blockDim.x) {
        s.x += a[p].x * b[p].x + a[p].y * b[p].y;
        s.y += a[p].x * b[p].y - a[p].y * b[p].x;
    }
    red[threadIdx.x] = s;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) red[threadIdx.x] = {red[threadIdx.x].x + red[threadIdx.x + k].x,
                                                 red[threadIdx.x].y + red[threadIdx.x + k].y};
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = red[0];
}

// v /= c (complex), c read from the device
__global__ void k_scale_inv(int npw, const double2 *c, int conj_c, double2 *v)
{
    double2 d = *c;
    if (conj_c) d.y = -d.y;
    const double den = d.x * d.x + d.y * d.y;
    const double2 inv = {d.x / den, -d.y / den};
    for (int p = blockIdx.x * blockDim.x + threadIdx.x; p < npw; p += gridDim.x * blockDim.x) {
        const double2 a = v[p];
        v[p] = {a.x * inv.x - a.y * inv.y, a.x * inv.y + a.y * inv.x};
    }
}

// ------------------------------------------- blocked Gram-Schmidt ---------
// Modified Gram-Schmidt in the reference's order (each vector loses its
// components along the earlier ones one after the other), arranged so that
// many vectors advance at once: k_mgs_update takes a range of finished rows
// out of every remaining vector (one CTA per vector, its elements in
// registers), k_mgs_panel finishes PANEL vectors in one cluster of PANEL CTAs
// (a vector each; the cluster barrier orders them).  The sequence of
// operations of each vector is that of the vector-by-vector loop.
// What bounds a projection is the read of one row by one SM (16 npw bytes) and
// one block reduction; with one CTA for all vectors in turn the eight-atom
// cell's step (48 new vectors on 48, 4600 plane waves) took 3400 of them in a
// row, here 48 + 6 x 16.
constexpr int GT = 512;          // threads per vector
constexpr int PANEL = 8;         // vectors per cluster

// sum of (x, y) over the block, the same value in every thread
__device__ __forceinline__ double2 block_sum(double2 s)
{
    __shared__ double2 part[GT / 32];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        s.x += __shfl_xor_sync(0xffffffffu, s.x, o);
        s.y += __shfl_xor_sync(0xffffffffu, s.y, o);
    }
    __syncthreads();                          // the previous sum has been read
    if ((threadIdx.x & 31) == 0) part[threadIdx.x >> 5] = s;
    __syncthreads();
    double2 r = part[0];
#pragma unroll
    for (int w = 1; w < GT / 32; w++) r = {r.x + part[w].x, r.y + part[w].y};
    return r;
}

// A vector of npw elements spread over the block: E elements per thread in
// registers (npw <= E GT), or, with E = 0, left in global memory.
template <int E> struct Vec {
    double2 v[E > 0 ? E : 1];
    double2 *g;
    int npw;
    __device__ __forceinline__ void open(double2 *p, int n)
    {
        g = p;
        npw = n;
#pragma unroll
        for (int e = 0; e < E; e++) {
            const int q = threadIdx.x + e * GT;
            v[e] = q < n ? p[q] : double2{0, 0};
        }
    }
    // v -= <row|v> row
    __device__ __forceinline__ void project(const double2 *row)
    {
        if constexpr (E > 0) {
            double2 r[E], s = {0, 0};
#pragma unroll
            for (int e = 0; e < E; e++) {
                const int q = threadIdx.x + e * GT;
                r[e] = q < npw ? row[q] : double2{0, 0};
            }
#pragma unroll
            for (int e = 0; e < E; e++) {
                s.x += r[e].x * v[e].x + r[e].y * v[e].y;
                s.y += r[e].x * v[e].y - r[e].y * v[e].x;
            }
            const double2 c = block_sum(s);
#pragma unroll
            for (int e = 0; e < E; e++) {
                v[e].x -= c.x * r[e].x - c.y * r[e].y;
                v[e].y -= c.x * r[e].y + c.y * r[e].x;
            }
        } else {
            double2 s = {0, 0};
            for (int q = threadIdx.x; q < npw; q += GT) {
                const double2 a = row[q], b = g[q];
                s.x += a.x * b.x + a.y * b.y;
                s.y += a.x * b.y - a.y * b.x;
            }
            const double2 c = block_sum(s);
            for (int q = threadIdx.x; q < npw; q += GT) {
                const double2 a = row[q];
                g[q].x -= c.x * a.x - c.y * a.y;
                g[q].y -= c.x * a.y + c.y * a.x;
            }
        }
    }
    __device__ __forceinline__ double norm() const
    {
        double2 s = {0, 0};
        if constexpr (E > 0) {
#pragma unroll
            for (int e = 0; e < E; e++) s.x += v[e].x * v[e].x + v[e].y * v[e].y;
        } else {
            for (int q = threadIdx.x; q < npw; q += GT) s.x += g[q].x * g[q].x + g[q].y * g[q].y;
        }
        return sqrt(block_sum(s).x);
    }
    __device__ __forceinline__ void store(double2 *out, double scale) const
    {
        if constexpr (E > 0) {
#pragma unroll
            for (int e = 0; e < E; e++) {
                const int q = threadIdx.x + e * GT;
                if (q < npw) out[q] = {v[e].x * scale, v[e].y * scale};
            }
        } else if (out != g || scale != 1.0) {
            for (int q = threadIdx.x; q < npw; q += GT) out[q] = {g[q].x * scale, g[q].y * scale};
        }
    }
};

// rows [lo[0], hi[0]) of V out of vector blockIdx.x of T (lo, hi on the device)
template <int E>
__global__ void __launch_bounds__(GT) k_mgs_update(int npw, const double2 *V, const int *lo, const int *hi, double2 *T)
{
    Vec<E> x;
    double2 *t = T + (size_t)blockIdx.x * npw;
    x.open(t, npw);
    const int a = *lo, b = *hi;
    for (int i = a; i < b; i++) x.project(V + (size_t)i * npw);
    x.store(t, 1.0);
}

// One cluster: vectors 0 .. nv - 1 (nv <= PANEL) of T orthonormalised in order
// and appended to V from row *count on; one whose norm is below 1e-8 is left
// out.  count_out: the new number of rows; kept: its flag per vector.
template <int E>
__global__ void __cluster_dims__(PANEL, 1, 1) __launch_bounds__(GT)
    k_mgs_panel(int npw, int nv, double2 *V, double2 *T, const int *count, int *count_out, int *kept)
{
    const int me = blockIdx.x;
    Vec<E> x;
    if (me < nv) x.open(T + (size_t)me * npw, npw);
    int row = *count;
    for (int j = 0; j < nv; j++) {
        if (me == j) {
            const double nrm = x.norm();
            const bool ok = !(nrm < 1e-8);
            if (ok) x.store(V + (size_t)row * npw, 1.0 / nrm);
            if (threadIdx.x == 0) kept[j] = ok ? 1 : 0;
        }
        // the row and its flag become visible to the cluster
        asm volatile("barrier.cluster.arrive.release;\n" ::: "memory");
        asm volatile("barrier.cluster.wait.acquire;\n" ::: "memory");
        const bool on = *(volatile int *)&kept[j] != 0;
        if (on && me > j && me < nv) x.project(V + (size_t)row * npw);
        row += on ? 1 : 0;
    }
    if (me == 0 && threadIdx.x == 0) *count_out = row;
}

template <int E>
int mgs_run(int nv, int npw, double2 *V, double2 *T, int nbasis, int *counts, int *kept, cudaStream_t st)
{
    // counts[0] = 0, counts[1] = nbasis, then one entry per panel
    if (nbasis > 0) k_mgs_update<E><<<nv, GT, 0, st>>>(npw, V, counts, counts + 1, T);
    int *cnt = counts + 1;
    for (int j0 = 0; j0 < nv; j0 += PANEL, cnt++) {
        const int n = std::min(PANEL, nv - j0);
        k_mgs_panel<E><<<PANEL, GT, 0, st>>>(npw, n, V, T + (size_t)j0 * npw, cnt, cnt + 1, kept + j0);
        if (j0 + n < nv)
            k_mgs_update<E><<<nv - j0 - n, GT, 0, st>>>(npw, V, cnt, cnt + 1, T + (size_t)(j0 + n) * npw);
    }
    SUB_CUDA(cudaGetLastError());
    return TCG_OK;
}

// number of ints mgs needs
size_t mgs_ints(int nv) { return 2 + (nv + PANEL - 1) / PANEL + (size_t)nv; }

// Orthonormalise the nv vectors T against the nbasis rows of V and one another
// and append them to V (see k_mgs_panel; V may be T when nbasis = 0 and no vector
// vanishes).  ints: mgs_ints(nv) device ints; *rows: the new number of rows.
int mgs(int nv, int npw, double2 *V, double2 *T, int nbasis, int *ints, int *rows, cudaStream_t st)
{
    const int np = (nv + PANEL - 1) / PANEL;
    const int init[2] = {0, nbasis};
    SUB_CUDA(cudaMemcpyAsync(ints, init, sizeof init, cudaMemcpyHostToDevice, st));
    int *kept = ints + 2 + np, rc;
    if (npw <= 2 * GT) rc = mgs_run<2>(nv, npw, V, T, nbasis, ints, kept, st);
    else if (npw <= 6 * GT) rc = mgs_run<6>(nv, npw, V, T, nbasis, ints, kept, st);
    else if (npw <= 10 * GT) rc = mgs_run<10>(nv, npw, V, T, nbasis, ints, kept, st);
    else rc = mgs_run<0>(nv, npw, V, T, nbasis, ints, kept, st);
    if (rc) return rc;
    SUB_CUDA(cudaMemcpyAsync(rows, ints + 1 + np, sizeof(int), cudaMemcpyDeviceToHost, st));
    SUB_CUDA(cudaStreamSynchronize(st));
    return TCG_OK;
}

// ------------------------------------------- eigenproblem of small matrices --
// General complex eigenproblem A X = X D of order n <= EIG_MAX in one CTA: the
// matrix in shared memory, Householder reduction to Hessenberg form, explicit
// single-shift QR (the iteration of the EISPACK routine COMQR2, Peters and
// Wilkinson 1970, with the deflation test of Ahues and Tisseur 1997; this test with
// its fallback for zero diagonals, the scaled Wilkinson shift and the exceptional
// shifts at iterations 10 and 20 of 30 follow LAPACK's ZLAHQR), triangular back
// substitution (its smallest pivot as in LAPACK's ZTREVC).  The rows of a sweep are a wavefront: the thread of column k
// carries its running element in a register, forms rotation k as soon as rotation
// k - 1 has arrived, and one barrier later every column applies it.  The columns
// (and Z, by the other half of the CTA) then need no barrier at all: a thread
// walks its own row.  What bounds it is the chain of some n^2 rotations (one
// reciprocal root and a barrier each).  An implicit sweep with two barriers and
// three roots per rotation took 13 ms at n = 96, this one 6.1; the library
// eigensolve, which splits the work between host and device, takes 15 to 37 ms.
constexpr int EIG_MAX = 112, ET = 256;   // threads 0-127: rows / columns of H; 128-255: rows of Z

__device__ __forceinline__ double2 zadd(double2 a, double2 b) { return {a.x + b.x, a.y + b.y}; }
__device__ __forceinline__ double2 zsub(double2 a, double2 b) { return {a.x - b.x, a.y - b.y}; }
__device__ __forceinline__ double2 zmul(double2 a, double2 b) { return {a.x * b.x - a.y * b.y, a.x * b.y + a.y * b.x}; }
__device__ __forceinline__ double2 zmulc(double2 a, double2 b) { return {a.x * b.x + a.y * b.y, a.x * b.y - a.y * b.x}; }  // conj(a) b
__device__ __forceinline__ double zabs1(double2 a) { return fabs(a.x) + fabs(a.y); }
__device__ __forceinline__ double zabs(double2 a) { return sqrt(a.x * a.x + a.y * a.y); }
// a / b without overflow of |b|^2 (Smith 1962)
__device__ __forceinline__ double2 zdiv(double2 a, double2 b)
{
    if (fabs(b.x) >= fabs(b.y)) {
        const double r = b.y / b.x, d = b.x + b.y * r;
        return {(a.x + a.y * r) / d, (a.y - a.x * r) / d};
    }
    const double r = b.x / b.y, d = b.x * r + b.y;
    return {(a.x * r + a.y) / d, (a.y * r - a.x) / d};
}
__device__ __forceinline__ double2 zsqrt(double2 a)
{
    if (a.x == 0.0 && a.y == 0.0) return {0.0, 0.0};
    const double t = sqrt(0.5 * (fabs(a.x) + zabs(a)));
    if (a.x >= 0.0) return {t, a.y / (2.0 * t)};
    return {fabs(a.y) / (2.0 * t), copysign(t, a.y)};
}

// A: n x n (column-major, overwritten work copy not needed afterwards); w [n]:
// eigenvalues; VR [n x n]: eigenvectors, unit norm, largest component real and
// positive; Z [n x n]: scratch; info: 0, or > 0 when the iteration did not
// converge or a result is not finite
__global__ void __launch_bounds__(ET) k_eig(int n, const double2 *A, double2 *w, double2 *VR, double2 *Z, int *info)
{
    extern __shared__ __align__(16) unsigned char eig_smem[];
    const int ld = n | 1, t = threadIdx.x, lane = t & 31, warp = t >> 5, r0 = t & 127;
    const bool zside = t >= 128;
    double2 *H = reinterpret_cast<double2 *>(eig_smem);     // H[r + ld c]
    double2 *vec = H + (size_t)ld * n;                       // [ET / 32][EIG_MAX] vectors
    __shared__ double red[ET / 32];
    __shared__ int ired[ET / 32];
    const double ulp = 2.220446049250313e-16, tiny = 2.2250738585072014e-308 / ulp * n;
    auto h = [&](int r, int c) -> double2 & { return H[r + ld * c]; };
    for (int i = t; i < n * n; i += ET) {
        h(i % n, i / n) = A[i];
        Z[i] = make_double2(i % n == i / n ? 1.0 : 0.0, 0.0);
    }
    __syncthreads();
    auto sum = [&](double x) {
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) x += __shfl_xor_sync(0xffffffffu, x, o);
        __syncthreads();
        if (lane == 0) red[warp] = x;
        __syncthreads();
        double s = 0;
#pragma unroll
        for (int i = 0; i < ET / 32; i++) s += red[i];
        return s;
    };
    // ---- Hessenberg: reflectors I - tau v v^H, v[k + 1] = 1, on rows and columns k + 1 ...
    for (int k = 0; k + 2 < n; k++) {
        const bool in = t > k + 1 && t < n;
        const double2 x = in ? h(t, k) : double2{0, 0}, al = h(k + 1, k);
        const double xn = sum(x.x * x.x + x.y * x.y);
        // nothing to annihilate (uniform).  Squares may underflow while x does not: then beta
        // is 0 and the results are not finite, which the caller takes to the library
        if (xn == 0.0 && al.y == 0.0 && !__syncthreads_or(zabs1(x) > 0.0)) continue;
        const double beta = -copysign(sqrt(al.x * al.x + al.y * al.y + xn), al.x);
        const double2 tau = {(beta - al.x) / beta, -al.y / beta};
        const double2 sc = zdiv(double2{1.0, 0.0}, double2{al.x - beta, al.y});
        __syncthreads();
        if (t == k + 1) vec[t] = {1.0, 0.0};
        if (in) vec[t] = zmul(sc, x);
        __syncthreads();
        // right: H <- H (I - tau v v^H) and Z <- Z (I - tau v v^H), thread = row
        if (r0 < n) {
            double2 *M = zside ? Z + r0 : H + r0;
            const int lm = zside ? n : ld;
            double2 a = {0, 0};
            for (int c = k + 1; c < n; c++) a = zadd(a, zmul(M[(size_t)lm * c], vec[c]));
            a = zmul(tau, a);
            for (int c = k + 1; c < n; c++)
                M[(size_t)lm * c] = zsub(M[(size_t)lm * c], zmul(a, double2{vec[c].x, -vec[c].y}));
        }
        __syncthreads();
        // left: H <- (I - conj(tau) v v^H) H, thread = column
        if (t >= k && t < n) {
            double2 a = {0, 0};
            for (int r = k + 1; r < n; r++) a = zadd(a, zmulc(vec[r], h(r, t)));
            a = zmulc(tau, a);
            for (int r = k + 1; r < n; r++) h(r, t) = zsub(h(r, t), zmul(vec[r], a));
        }
        __syncthreads();
        if (t > k + 1 && t < n) h(t, k) = {0, 0};
        __syncthreads();
    }
    // ---- QR iteration
    int fail = 0, i = n - 1, its = 0;
    const int maxit = 40 * (n > 10 ? n : 10);
    for (int total = 0; i >= 0; total++) {
        if (total > maxit) {
            fail = 1;
            break;
        }
        // largest k <= i whose subdiagonal element is negligible (0: none)
        int k = 0;
        if (t >= 1 && t <= i) {
            const double2 s = h(t, t - 1);
            bool small = zabs1(s) <= tiny;
            if (!small) {
                double tst = zabs1(h(t - 1, t - 1)) + zabs1(h(t, t));
                if (tst == 0.0) {
                    if (t >= 2) tst += zabs1(h(t - 1, t - 2));
                    if (t + 1 <= i) tst += zabs1(h(t + 1, t));
                }
                if (zabs1(s) <= ulp * tst) {
                    const double p = zabs1(s), q = zabs1(h(t - 1, t)), d = zabs1(h(t, t)), e = zabs1(zsub(h(t - 1, t - 1), h(t, t)));
                    const double ab = fmax(p, q), ba = fmin(p, q), aa = fmax(d, e), bb = fmin(d, e), q2 = aa + ab;
                    small = ba * (ab / q2) <= fmax(tiny, ulp * (bb * (aa / q2)));
                }
            }
            if (small) k = t;
        }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) k = max(k, __shfl_xor_sync(0xffffffffu, k, o));
        __syncthreads();
        if (lane == 0) ired[warp] = k;
        __syncthreads();
        int l = 0;
#pragma unroll
        for (int q = 0; q < ET / 32; q++) l = max(l, ired[q]);
        if (l > 0 && t == 0) h(l, l - 1) = {0, 0};
        if (l >= i) {
            i--;
            its = 0;
            __syncthreads();
            continue;
        }
        its++;
        // shift
        double2 sh;
        if (its % 30 == 10) {
            sh = h(l, l);
            sh.x += 0.75 * fabs(h(l + 1, l).x) + 0.75 * fabs(h(l + 1, l).y);
        } else if (its % 30 == 20) {
            sh = h(i, i);
            sh.x += 0.75 * fabs(h(i, i - 1).x) + 0.75 * fabs(h(i, i - 1).y);
        } else {
            sh = h(i, i);
            const double2 u = zmul(zsqrt(h(i - 1, i)), zsqrt(h(i, i - 1)));
            double s = zabs1(u);
            if (s != 0.0) {
                const double2 d = zsub(h(i - 1, i - 1), sh), x = {0.5 * d.x, 0.5 * d.y};
                const double sx = zabs1(x);
                s = fmax(s, sx);
                const double2 xs = {x.x / s, x.y / s}, us = {u.x / s, u.y / s};
                double2 y = zsqrt(zadd(zmul(xs, xs), zmul(us, us)));
                y = {s * y.x, s * y.y};
                if (sx > 0.0 && (x.x / sx) * y.x + (x.y / sx) * y.y < 0.0) y = {-y.x, -y.y};
                sh = zsub(sh, zmul(u, zdiv(u, zadd(x, y))));
            }
        }
        __syncthreads();                                      // the shift's elements have been read
        // rows: G_k (k = l ... i - 1) on rows k, k + 1 of H - sh, thread = column; p = the running
        // element of row k.  Thread k forms G_k = 1/r [conj(a) conj(b); -b a] from its column.
        double2 p = {0, 0};
        if (t >= l && t < n) p = h(l, t);
        if (t == l) p = zsub(p, sh);
        for (int k2 = l; k2 < i; k2++) {
            double2 q = {0, 0};
            if (t >= k2 && t < n) q = h(k2 + 1, t);
            if (t == k2 + 1) q = zsub(q, sh);
            if (t == k2) {
                double2 a = p, b = q;
                double n2 = a.x * a.x + a.y * a.y + (b.x * b.x + b.y * b.y), s = 1.0;
                if (!(n2 > 1e-280 && n2 < 1e280)) {
                    s = fmax(fmax(fabs(a.x), fabs(a.y)), fmax(fabs(b.x), fabs(b.y)));
                    if (s > 0.0 && isfinite(s)) {
                        a = {a.x / s, a.y / s};
                        b = {b.x / s, b.y / s};
                    } else {
                        a = {1.0, 0.0};
                        b = {0.0, 0.0};
                    }
                    n2 = a.x * a.x + a.y * a.y + (b.x * b.x + b.y * b.y);
                }
                const double ir = rsqrt(n2);
                vec[k2] = {a.x * ir, a.y * ir};
                vec[EIG_MAX + k2] = {b.x * ir, b.y * ir};
                h(k2, k2) = {s * (n2 * ir), 0.0};
                h(k2 + 1, k2) = {0, 0};
            }
            __syncthreads();
            if (t > k2 && t < n) {
                const double2 ca = vec[k2], cb = vec[EIG_MAX + k2];
                h(k2, t) = zadd(zmulc(ca, p), zmulc(cb, q));
                p = zsub(zmul(ca, q), zmul(cb, p));
            }
        }
        if (t >= i && t < n) h(i, t) = p;
        __syncthreads();
        // columns: G_k^H on columns k, k + 1 of H (rows 0 ... i) and Z, thread = row; x = the
        // running element of column k, the columns after it on their way
        {
            const int rows = zside ? n : i + 1;
            if (r0 < rows) {
                double2 *M = zside ? Z + r0 : H + r0;
                const size_t lm = zside ? n : ld;
                const int kb = zside ? l : max(l, r0 - 1);
                double2 x = M[lm * kb], y[4];
                int k2 = kb;
                const bool dg = !zside && r0 >= l;
                auto step = [&](double2 yk) {
                    const double2 ca = vec[k2], cb = vec[EIG_MAX + k2];
                    double2 f = zadd(zmul(x, ca), zmul(yk, cb));
                    if (dg && k2 == r0) f = zadd(f, sh);
                    M[lm * k2] = f;
                    x = zsub(zmulc(ca, yk), zmulc(cb, x));
                    k2++;
                };
#pragma unroll
                for (int m = 0; m < 4; m++)
                    if (kb + 1 + m <= i) y[m] = M[lm * (kb + 1 + m)];
                while (k2 + 4 <= i) {
#pragma unroll
                    for (int m = 0; m < 4; m++) {
                        const double2 yk = y[m];
                        if (k2 + 5 <= i) y[m] = M[lm * (k2 + 5)];
                        step(yk);
                    }
                }
#pragma unroll
                for (int m = 0; m < 4; m++)
                    if (k2 < i) step(y[m]);
                if (dg && r0 == i) x = zadd(x, sh);
                M[lm * i] = x;
            }
        }
        __syncthreads();
    }
    // ---- eigenvalues and vectors
    if (!fail) {
        if (t < n) w[t] = h(t, t);
        double2 *x = vec + warp * EIG_MAX;
        bool bad = false;
        for (int k = warp; k < n; k += ET / 32) {
            const double2 lam = h(k, k);
            const double smin = fmax(ulp * zabs1(lam), tiny);
            for (int r = lane; r <= k; r += 32) x[r] = r == k ? double2{1.0, 0.0} : double2{-h(r, k).x, -h(r, k).y};
            __syncwarp();
            for (int j = k - 1; j >= 0; j--) {
                double2 d = zsub(h(j, j), lam);
                if (zabs1(d) < smin) d = {smin, 0.0};
                const double2 xj = zdiv(x[j], d);
                __syncwarp();
                if (lane == 0) x[j] = xj;
                for (int r = lane; r < j; r += 32) x[r] = zsub(x[r], zmul(xj, h(r, j)));
                __syncwarp();
            }
            double2 v[(EIG_MAX + 31) / 32];
            double nrm = 0, big = -1.0;
            int at = 0;
#pragma unroll
            for (int e = 0; e < (EIG_MAX + 31) / 32; e++) {
                const int r = lane + 32 * e;
                v[e] = {0, 0};
                if (r < n) {
                    for (int j = 0; j <= k; j++) v[e] = zadd(v[e], zmul(Z[r + (size_t)n * j], x[j]));
                    const double m = v[e].x * v[e].x + v[e].y * v[e].y;
                    nrm += m;
                    if (m > big) { big = m; at = r; }
                }
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                nrm += __shfl_xor_sync(0xffffffffu, nrm, o);
                const double ob = __shfl_xor_sync(0xffffffffu, big, o);
                const int oa = __shfl_xor_sync(0xffffffffu, at, o);
                if (ob > big || (ob == big && oa < at)) { big = ob; at = oa; }
            }
            double2 top = {0, 0};
#pragma unroll
            for (int e = 0; e < (EIG_MAX + 31) / 32; e++)
                if (lane + 32 * e == at) top = v[e];
            top.x = __shfl_sync(0xffffffffu, top.x, at & 31);
            top.y = __shfl_sync(0xffffffffu, top.y, at & 31);
            const double nn = sqrt(nrm), bt = sqrt(big);
            const double2 f = {top.x / bt / nn, -top.y / bt / nn};
            bad = bad || !isfinite(f.x) || !isfinite(f.y) || !isfinite(nn);
#pragma unroll
            for (int e = 0; e < (EIG_MAX + 31) / 32; e++) {
                const int r = lane + 32 * e;
                double2 o = zmul(v[e], f);
                if (r == at) o.y = 0.0;
                if (r < n) VR[r + (size_t)n * k] = o;
            }
            __syncwarp();
        }
        if (bad) fail = 2;
    }
    fail = __syncthreads_or(fail);
    if (t == 0) *info = fail;
}

// make_a_new_trial_vector (diagonalization_utils.cpp:165-211) for vector b
// of a block, one CTA each: with the kinetic expectation
// t = <phi| |k+G|^2 |phi> / <phi|phi> and x = |k+G|^2 / t, the Payne
// preconditioner K(x) = (27 + 18x + 12x^2 + 8x^3) / (27 + 18x + 12x^2 + 8x^3 + 16x^4)
// gives dst = -K (H phi - e phi), normalised, or zero when its norm is below 1e-8
__global__ void k_precondition(int npw, const double *kg2, const double2 *phi, const double2 *h1, const double2 *h2,
                               const double2 *h3, const double2 *eig, double2 *dst)
{
    __shared__ double ra[256], rb[256];
    const size_t off = (size_t)blockIdx.x * npw;
    double a = 0, n = 0;
    for (int p = threadIdx.x; p < npw; p += blockDim.x) {
        const double2 v = phi[off + p];
        const double q = v.x * v.x + v.y * v.y;
        a += kg2[p] * q;
        n += q;
    }
    ra[threadIdx.x] = a;
    rb[threadIdx.x] = n;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) {
            ra[threadIdx.x] += ra[threadIdx.x + k];
            rb[threadIdx.x] += rb[threadIdx.x + k];
        }
        __syncthreads();
    }
    const double kin = ra[0] / rb[0];
    const double2 e = eig[blockIdx.x];
    __syncthreads();
    double s = 0;
    for (int p = threadIdx.x; p < npw; p += blockDim.x) {
        const double x = kg2[p] / kin;
        const double c = (27 + x * (18 + x * (12 + x * 8))) / (27 + x * (18 + x * (12 + x * (8 + x * 16))));
        const double2 v = phi[off + p];
        double2 r = {-(e.x * v.x - e.y * v.y), -(e.x * v.y + e.y * v.x)};
        if (h1) r = {r.x + h1[off + p].x, r.y + h1[off + p].y};
        if (h2) r = {r.x + h2[off + p].x, r.y + h2[off + p].y};
        if (h3) r = {r.x + h3[off + p].x, r.y + h3[off + p].y};
        const double2 o = {-c * r.x, -c * r.y};
        dst[off + p] = o;
        s += o.x * o.x + o.y * o.y;
    }
    ra[threadIdx.x] = s;
    __syncthreads();
    for (int k = blockDim.x / 2; k > 0; k >>= 1) {
        if (threadIdx.x < k) ra[threadIdx.x] += ra[threadIdx.x + k];
        __syncthreads();
    }
    const double nrm = sqrt(ra[0]);
    const double scale = nrm < 1e-8 ? 0.0 : 1.0 / nrm;
    for (int p = threadIdx.x; p < npw; p += blockDim.x) {
        const double2 o = dst[off + p];
        dst[off + p] = {o.x * scale, o.y * scale};
    }
}

} // namespace

extern "C" int tcg_davidson_expand(int32_t nbasis, int32_t nblock, int32_t npw, void *V, const void *phi,
                                   const void *H1phi, const void *H2phi, const void *H3phi, const double *kG2,
                                   const double *eig_ref, int32_t *nbasis_out, void *stream)
{
    if (nbasis < 0 || nblock < 0 || npw < 1 || !V || !nbasis_out || (nblock > 0 && (!phi || !kG2 || !eig_ref)) ||
        (nblock > 0 && !H1phi && !H2phi && !H3phi))
        return fail(TCG_ERR_ARG, "bad Davidson expansion arguments");
    *nbasis_out = nbasis;
    if (nblock == 0) return TCG_OK;
    cudaStream_t st = (cudaStream_t)stream;
    Scratch S(st);
    int rc;
    const size_t nt = (size_t)nblock * npw;
    if ((rc = S.reserve(Scratch::part(nt * sizeof(double2)) + Scratch::part(nblock * sizeof(double2)) +
                        Scratch::part(mgs_ints(nblock) * sizeof(int)))))
        return rc;
    double2 *T = S.get<double2>(nt), *de = S.get<double2>(nblock);
    int *ints = S.get<int>(mgs_ints(nblock));
    SUB_CUDA(cudaMemcpyAsync(de, eig_ref, nblock * sizeof(double2), cudaMemcpyHostToDevice, st));
    k_precondition<<<nblock, 256, 0, st>>>(npw, kG2, (const double2 *)phi, (const double2 *)H1phi,
                                           (const double2 *)H2phi, (const double2 *)H3phi, de, T);
    SUB_CUDA(cudaGetLastError());
    // Gram_Schmidt of each new vector against the whole current basis, the new
    // vectors of this block included; a vector below norm 1e-8 is dropped
    // (diagonalization_davidson.cpp:297-318)
    int rows = 0;
    if ((rc = mgs(nblock, npw, (double2 *)V, T, nbasis, ints, &rows, st))) return rc;
    *nbasis_out = rows;
    return TCG_OK;
}

extern "C" int tcg_subspace_ritz(int32_t ndim, int32_t npw, int32_t nout, int32_t biortho, const void *V,
                                 const void *Vref, const void *H1V, const void *H2V, const void *H3V, double *eig_out,
                                 double *e_out, void *V_out, void *Vl_out, void *stream)
{
    if (ndim < 1 || npw < 1 || nout < 0 || nout > ndim) return fail(TCG_ERR_ARG, "bad subspace sizes");
    if (!V || !eig_out || (!H1V && !H2V && !H3V)) return fail(TCG_ERR_ARG, "null argument");
    if (nout > 0 && !V_out) return fail(TCG_ERR_ARG, "V_out is NULL");
    if (!Vref) Vref = V;
    Handles *hd;
    int rc = handles(&hd);
    if (rc) return rc;
    cudaStream_t st = (cudaStream_t)stream;
    SUB_BLAS(cublasSetStream(hd->blas, st));
    SUB_SOLV(cusolverDnSetStream(hd->solver, st));
    Scratch S(st);
    const size_t nn = (size_t)ndim * ndim;
    const void *HV[3] = {H1V, H2V, H3V};
    // workspace size of the LU (the matrix argument is not read)
    int lwork = 0;
    SUB_SOLV(cusolverDnZgetrf_bufferSize(hd->solver, ndim, ndim, nullptr, ndim, &lwork));
    if ((rc = S.reserve(9 * Scratch::part(nn * sizeof(double2)) + Scratch::part(ndim * sizeof(double2)) +
                        Scratch::part(3 * (size_t)ndim * sizeof(double2)) + Scratch::part((size_t)lwork * sizeof(double2)) +
                        2 * Scratch::part(ndim * sizeof(int)) + Scratch::part(64 * sizeof(int)))))
        return rc;
    double2 *Hn[3] = {nullptr, nullptr, nullptr};
    for (int n = 0; n < 3; n++)
        if (HV[n]) Hn[n] = S.get<double2>(nn);
    double2 *H = S.get<double2>(nn), *A = S.get<double2>(nn), *VR = S.get<double2>(nn), *X = S.get<double2>(nn);
    double2 *Xinv = S.get<double2>(nn), *XL = S.get<double2>(nn), *W = S.get<double2>(ndim);
    double2 *E = S.get<double2>(3 * (size_t)ndim);
    void *lw = S.get<double2>(lwork);
    int *dinfo = S.get<int>(64), *dperm = S.get<int>(ndim), *ipiv = S.get<int>(ndim);
    // H_n,sub(i, j) = <Vref_i | H_n V_j>   (diagonalization_davidson.cpp:462-475)
    const cuDoubleComplex one = make_cuDoubleComplex(1, 0), zero = make_cuDoubleComplex(0, 0);
    for (int n = 0; n < 3; n++)
        if (HV[n])
            SUB_BLAS(cublasZgemm(hd->blas, CUBLAS_OP_C, CUBLAS_OP_N, ndim, ndim, npw, &one, (const cuDoubleComplex *)Vref,
                                 npw, (const cuDoubleComplex *)HV[n], npw, &zero, (cuDoubleComplex *)Hn[n], ndim));
    k_add3<<<(unsigned)((nn + 255) / 256), 256, 0, st>>>((int)nn, Hn[0], Hn[1], Hn[2], H);
    SUB_CUDA(cudaGetLastError());
    // H_sub X = X D (ComplexEigenSolver, :479-486): in one CTA up to order EIG_MAX (what its
    // shared memory holds), by cuSOLVER beyond and where that iteration does not converge
    int info = -1;
    std::vector<double2> w(ndim);
    if (ndim <= EIG_MAX) {
        const size_t sm = ((size_t)(ndim | 1) * ndim + ET / 32 * EIG_MAX) * sizeof(double2);
        SUB_CUDA(cudaFuncSetAttribute(k_eig, cudaFuncAttributeMaxDynamicSharedMemorySize, 227 * 1024 - 256));
        k_eig<<<1, ET, sm, st>>>(ndim, H, W, VR, Xinv, dinfo);
        SUB_CUDA(cudaGetLastError());
        SUB_CUDA(cudaMemcpyAsync(&info, dinfo, sizeof(int), cudaMemcpyDeviceToHost, st));
        SUB_CUDA(cudaMemcpyAsync(w.data(), W, ndim * sizeof(double2), cudaMemcpyDeviceToHost, st));
        SUB_CUDA(cudaStreamSynchronize(st));
    }
    if (info != 0) {
        size_t dws = 0, hws = 0;
        SUB_SOLV(cusolverDnXgeev_bufferSize(hd->solver, hd->params, CUSOLVER_EIG_MODE_NOVECTOR, CUSOLVER_EIG_MODE_VECTOR,
                                            ndim, CUDA_C_64F, A, ndim, CUDA_C_64F, W, CUDA_C_64F, nullptr, ndim, CUDA_C_64F,
                                            VR, ndim, CUDA_C_64F, &dws, &hws));
        Scratch S2(st);
        if ((rc = S2.reserve(Scratch::part(dws)))) return rc;
        std::vector<unsigned char> hwork(std::max<size_t>(hws, 16));
        SUB_CUDA(cudaMemcpyAsync(A, H, nn * sizeof(double2), cudaMemcpyDeviceToDevice, st));
        SUB_SOLV(cusolverDnXgeev(hd->solver, hd->params, CUSOLVER_EIG_MODE_NOVECTOR, CUSOLVER_EIG_MODE_VECTOR, ndim,
                                 CUDA_C_64F, A, ndim, CUDA_C_64F, W, CUDA_C_64F, nullptr, ndim, CUDA_C_64F, VR, ndim,
                                 CUDA_C_64F, S2.get<char>(dws), dws, hwork.data(), hws, dinfo));
        SUB_CUDA(cudaMemcpyAsync(&info, dinfo, sizeof(int), cudaMemcpyDeviceToHost, st));
        SUB_CUDA(cudaMemcpyAsync(w.data(), W, ndim * sizeof(double2), cudaMemcpyDeviceToHost, st));
        SUB_CUDA(cudaStreamSynchronize(st));
        if (info != 0) return fail(TCG_ERR_NUMERIC, "diagonalization of H_subspace failed");
    }
    // sort by the real part, ascending (sort_eigen, diagonalization_utils.cpp:82-119)
    std::vector<int> perm(ndim);
    std::iota(perm.begin(), perm.end(), 0);
    std::stable_sort(perm.begin(), perm.end(), [&](int a, int b) { return w[a].x < w[b].x; });
    for (int i = 0; i < ndim; i++) {
        eig_out[2 * i] = w[perm[i]].x;
        eig_out[2 * i + 1] = w[perm[i]].y;
    }
    SUB_CUDA(cudaMemcpyAsync(dperm, perm.data(), ndim * sizeof(int), cudaMemcpyHostToDevice, st));
    k_permute_cols<<<ndim, 128, 0, st>>>(ndim, dperm, VR, X);
    // X^-1 by LU (eigenvectors.inverse(), :494); left eigenvectors (X^-1)^H
    SUB_CUDA(cudaMemcpyAsync(A, X, nn * sizeof(double2), cudaMemcpyDeviceToDevice, st));
    SUB_SOLV(cusolverDnZgetrf(hd->solver, ndim, ndim, (cuDoubleComplex *)A, ndim, (cuDoubleComplex *)lw, ipiv, dinfo));
    k_identity<<<ndim, 128, 0, st>>>(ndim, Xinv);
    SUB_SOLV(cusolverDnZgetrs(hd->solver, CUBLAS_OP_N, ndim, ndim, (const cuDoubleComplex *)A, ndim, ipiv,
                              (cuDoubleComplex *)Xinv, ndim, dinfo));
    SUB_CUDA(cudaMemcpyAsync(&info, dinfo, sizeof(int), cudaMemcpyDeviceToHost, st));
    k_adjoint<<<ndim, 128, 0, st>>>(ndim, Xinv, XL);
    SUB_CUDA(cudaGetLastError());
    // Ritz vectors V X and left vectors Vref X_left (:497-530)
    if (nout > 0) {
        SUB_BLAS(cublasZgemm(hd->blas, CUBLAS_OP_N, CUBLAS_OP_N, npw, nout, ndim, &one, (const cuDoubleComplex *)V, npw,
                             (const cuDoubleComplex *)X, ndim, &zero, (cuDoubleComplex *)V_out, npw));
        if (Vl_out)
            SUB_BLAS(cublasZgemm(hd->blas, CUBLAS_OP_N, CUBLAS_OP_N, npw, nout, ndim, &one, (const cuDoubleComplex *)Vref,
                                 npw, (const cuDoubleComplex *)XL, ndim, &zero, (cuDoubleComplex *)Vl_out, npw));
    }
    // energies diag(L^H H_n,sub X), L = X_left for BITC, X otherwise (:583-596)
    if (e_out && nout > 0) {
        for (int n = 0; n < 3; n++)
            if (Hn[n]) k_diag_form<<<nout, 256, 0, st>>>(ndim, nout, biortho ? XL : X, Hn[n], X, E + (size_t)n * ndim);
        SUB_CUDA(cudaGetLastError());
        std::vector<double2> e(3 * (size_t)ndim, make_double2(0, 0));
        for (int n = 0; n < 3; n++)
            if (Hn[n]) SUB_CUDA(cudaMemcpyAsync(e.data() + (size_t)n * ndim, E + (size_t)n * ndim, nout * sizeof(double2),
                                                cudaMemcpyDeviceToHost, st));
        SUB_CUDA(cudaStreamSynchronize(st));
        for (int n = 0; n < 3; n++)
            for (int i = 0; i < nout; i++) {
                e_out[2 * ((size_t)n * nout + i)] = e[(size_t)n * ndim + i].x;
                e_out[2 * ((size_t)n * nout + i) + 1] = e[(size_t)n * ndim + i].y;
            }
    }
    SUB_CUDA(cudaStreamSynchronize(st));
    if (info != 0) return fail(TCG_ERR_NUMERIC, "eigenvector matrix of H_subspace is singular");
    return TCG_OK;
}

extern "C" int tcg_gram_schmidt(int32_t nvec, int32_t npw, void *V, void *Vl, void *stream)
{
    if (nvec < 0 || npw < 1 || !V) return fail(TCG_ERR_ARG, "bad Gram-Schmidt arguments");
    cudaStream_t st = (cudaStream_t)stream;
    if (nvec == 0) return TCG_OK;
    Scratch S(st);
    int rc;
    double2 *v = (double2 *)V, *l = (double2 *)Vl;
    if (!l) {
        if ((rc = S.reserve(Scratch::part(mgs_ints(nvec) * sizeof(int))))) return rc;
        int rows = 0;
        if ((rc = mgs(nvec, npw, v, v, 0, S.get<int>(mgs_ints(nvec)), &rows, st))) return rc;
        if (rows < nvec) return fail(TCG_ERR_NUMERIC, "Linear independence breaks in block-Davidson algorithm.");
        return TCG_OK;
    }
    if ((rc = S.reserve(Scratch::part(nvec * sizeof(double2))))) return rc;
    double2 *c = S.get<double2>(nvec);
    for (int j = 0; j < nvec; j++) {
        double2 *tj = v + (size_t)j * npw;
        // |j> -= <ref_i|j> |i>, i < j  (Gram_Schmidt / Gram_Schmidt_biortho, utils:7-77)
        k_gs_project<<<1, 256, 0, st>>>(npw, j, l, v, tj);
        k_dotc<<<1, 256, 0, st>>>(npw, tj, tj, c + j);            // |j|^2
        SUB_CUDA(cudaGetLastError());
        double2 nrm2;
        SUB_CUDA(cudaMemcpyAsync(&nrm2, c + j, sizeof(double2), cudaMemcpyDeviceToHost, st));
        SUB_CUDA(cudaStreamSynchronize(st));
        const double nrm = std::sqrt(nrm2.x);
        if (nrm < 1e-10) return fail(TCG_ERR_NUMERIC, "Linear independence breaks in block-Davidson algorithm.");
        double2 hn = make_double2(nrm, 0.0);
        SUB_CUDA(cudaMemcpyAsync(c + j, &hn, sizeof(double2), cudaMemcpyHostToDevice, st));
        k_scale_inv<<<8, 256, 0, st>>>(npw, c + j, 0, tj);
        double2 *lj = l + (size_t)j * npw;
        // <j| -= <j|i> <i|, then <j|j> = 1 by dividing the left vector by conj(<l_j|v_j>)
        k_gs_project<<<1, 256, 0, st>>>(npw, j, v, l, lj);
        k_dotc<<<1, 256, 0, st>>>(npw, lj, tj, c + j);
        double2 cc;
        SUB_CUDA(cudaMemcpyAsync(&cc, c + j, sizeof(double2), cudaMemcpyDeviceToHost, st));
        SUB_CUDA(cudaStreamSynchronize(st));
        if (std::sqrt(cc.x * cc.x + cc.y * cc.y) < 1e-10)
            return fail(TCG_ERR_NUMERIC, "Linear independence breaks in block-Davidson algorithm.");
        k_scale_inv<<<8, 256, 0, st>>>(npw, c + j, 1, lj);
        SUB_CUDA(cudaGetLastError());
    }
    SUB_CUDA(cudaStreamSynchronize(st));
    return TCG_OK;
}
