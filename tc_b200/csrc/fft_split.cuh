// fft_split.cuh -- whole 3-D transforms of lists of grids (natural order, x fastest,
// on both sides) on the compiled cubic sizes, in split lines (split.cuh): orbitals
// onto the grid, accumulators back onto the sphere, the per-state fields.  The
// generic forms (passes.cuh) make one shared-memory sweep and one barrier per radix.
// The passes move each grid four times; where there are enough grids to fill the
// device memory traffic bounds them (gradient tables on 40^3: 2.74 -> 1.52 ms), for a
// few grids the launch and one line's latency do (5 us a pass).
#pragma once
#include "terms.cuh"
#include "split.cuh"

namespace tcg {
namespace sl {

template <typename V, class S> constexpr size_t smem_xy_io() { return sizeof(V) * 2 * (size_t)S::N * S::PAD; }
template <typename V, class S> constexpr size_t smem_z_io() { return sizeof(V) * (size_t)S::N * 32; }

// XY transform in place, one plane per CTA; the plane turns between the x-fastest
// order in memory and the y-fastest order of the G side in shared memory
template <typename T, class S, int DIR>
__global__ void __launch_bounds__(S::THREADS, ctas_for(S::THREADS, sizeof(T) == 4 ? 64 : 112)) k_xy_io(GridDesc g, GridRefs grids)
{
    using V = typename C2<T>::t;
    constexpr int N = S::N, A = S::A, B = S::B, PS = S::N * S::PAD, PAD = S::PAD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *b0 = reinterpret_cast<V *>(smem_raw), *b1 = b0 + PS;
    const int t = threadIdx.x / S::LP, l = threadIdx.x % S::LP;
    const bool on = S::LP == N || l < N;
    V *grid = reinterpret_cast<V *>(grids[blockIdx.y]) + (size_t)blockIdx.x * N * N + l;
    if constexpr (DIR < 0) {
        Tw<V, B> tw;
        tw.load(g, t);
        V u[B], v[A];
        if (on) {
#pragma unroll
            for (int m = 0; m < B; m++) u[m] = grid[(t + A * m) * N];
        }
        plane_fwd<V, S>(b0, b1, t, l, u, tw, v);
        if (on && t < B) {
#pragma unroll
            for (int m = 0; m < A; m++) b1[l * PAD + t + B * m] = v[m];      // row ky = l
        }
        __syncthreads();
        if (on) {
#pragma unroll
            for (int m = 0; m < B; m++) grid[(t + A * m) * N] = b1[(t + A * m) * PAD + l];
        }
    } else {
        Tw<V, A> tw;
        tw.load(g, t < B ? t : 0);
        V u[A], v[B];
        if (on) {
#pragma unroll
            for (int m = 0; m < B; m++) b1[(t + A * m) * PAD + l] = grid[(t + A * m) * N];
        }
        __syncthreads();
        if (on && t < B) {
#pragma unroll
            for (int m = 0; m < A; m++) u[m] = b1[l * PAD + t + B * m];
        }
        plane_inv<V, S>(b0, b1, t, l, u, tw, v);
        if (on) {
#pragma unroll
            for (int m = 0; m < B; m++) grid[(t + A * m) * N] = v[m];
        }
    }
}

// Z transform of 32 pencils per CTA.  forward: u[m] at z = t + A m, t < A -> v[m] at z = t + B m, t < B
template <typename V, class S>
__device__ __forceinline__ void z_fwd(V *E, int t, const GridDesc &g, V (&u)[S::B], V (&v)[S::A])
{
    Tw<V, S::B> tw;
    tw.load(g, t);
    step1<V, S::B, -1>(u, tw);
    put<V, S::A, S::B>(E, 32, t, u);
    __syncthreads();
    if (t < S::B) step2<V, S::A, S::B, -1>(E, 32, t, v);
}
// inverse: u[m] at z = t + B m, t < B -> v[m] at z = t + A m, t < A
template <typename V, class S>
__device__ __forceinline__ void z_inv(V *E, int t, const GridDesc &g, V (&u)[S::A], V (&v)[S::B])
{
    if (t < S::B) {
        Tw<V, S::A> tw;
        tw.load(g, t);
        step1<V, S::A, +1>(u, tw);
        put<V, S::B, S::A>(E, 32, t, u);
    }
    __syncthreads();
    step2<V, S::B, S::A, +1>(E, 32, t, v);
}

template <typename T, class S, int DIR>
__global__ void __launch_bounds__(S::ZTHREADS, ctas_for(S::ZTHREADS, sizeof(T) == 4 ? 48 : 80)) k_z_io(GridDesc g, GridRefs grids, T scale)
{
    using V = typename C2<T>::t;
    constexpr int N = S::N, A = S::A, B = S::B;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x / 32, cl = threadIdx.x % 32, c = blockIdx.x * 32 + cl;
    V *E = reinterpret_cast<V *>(smem_raw) + cl;
    const bool act = c < N * N;
    V *grid = reinterpret_cast<V *>(grids[blockIdx.y]) + c;
    V f[B], b[A];                                // A threads x B values, B threads x A values
    if constexpr (DIR < 0) {
#pragma unroll
        for (int m = 0; m < B; m++) f[m] = act ? grid[(t + A * m) * N * N] : czero<V>();
        z_fwd<V, S>(E, t, g, f, b);
        if (act && t < B) {
#pragma unroll
            for (int m = 0; m < A; m++) grid[(t + B * m) * N * N] = cscale(b[m], scale);
        }
    } else {
        if (t < B) {
#pragma unroll
            for (int m = 0; m < A; m++) b[m] = act ? grid[(t + B * m) * N * N] : czero<V>();
        }
        z_inv<V, S>(E, t, g, b, f);
        if (act) {
#pragma unroll
            for (int m = 0; m < B; m++) grid[(t + A * m) * N * N] = cscale(f[m], scale);
        }
    }
}

// the Z part of sphere -> grid: k_sphere_z's loads
template <typename T, class S>
__global__ void __launch_bounds__(S::ZTHREADS, ctas_for(S::ZTHREADS, sizeof(T) == 4 ? 64 : 96))
    k_sphere_io(GridDesc g, const SphereItem *items, const double *recip)
{
    using V = typename C2<T>::t;
    constexpr int N = S::N, A = S::A, B = S::B;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x / 32, cl = threadIdx.x % 32, c = blockIdx.x * 32 + cl;
    V *E = reinterpret_cast<V *>(smem_raw) + cl;
    const bool act = c < N * N;
    const SphereItem &it = items[blockIdx.y];
    V u[A], v[B];
    if (t < B) {
#pragma unroll
        for (int m = 0; m < A; m++) u[m] = act ? sphere_value<V>(g, it, recip, c, t + B * m) : czero<V>();
    }
    z_inv<V, S>(E, t, g, u, v);
    if (act) {
        V *out = reinterpret_cast<V *>(it.out) + c;
#pragma unroll
        for (int m = 0; m < B; m++) out[(size_t)(t + A * m) * N * N] = v[m];
    }
}

// the Z part of grid -> sphere: h[ip] += fac * grid(G)
template <class S>
__global__ void __launch_bounds__(S::ZTHREADS, ctas_for(S::ZTHREADS, 96)) k_gather_io(GridDesc g, const GatherItem *items)
{
    using V = double2;
    constexpr int N = S::N, A = S::A, B = S::B;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    const int t = threadIdx.x / 32, cl = threadIdx.x % 32, c = blockIdx.x * 32 + cl;
    V *E = reinterpret_cast<V *>(smem_raw) + cl;
    const bool act = c < N * N;
    const GatherItem &it = items[blockIdx.y];
    V u[B], v[A];
#pragma unroll
    for (int m = 0; m < B; m++) u[m] = act ? it.grid[(size_t)(t + A * m) * N * N + c] : czero<V>();
    z_fwd<V, S>(E, t, g, u, v);
    if (act && t < B) {
#pragma unroll
        for (int m = 0; m < A; m++) {
            const int ip = it.inv[(size_t)(t + B * m) * N * N + c];
            if (ip >= 0) it.h[ip] = cadd(it.h[ip], cmul(v[m], it.fac));
        }
    }
}

} // namespace sl
} // namespace tcg
