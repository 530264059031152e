// cube.cuh -- hf2x with the whole pair on chip, for work grids that fit one
// CTA's shared memory.
//
//   sum_q,i f phi_q(r) IFFT[ v(k - q + G) FFT[conj(phi_q) psi_k] ]
//
// One CTA takes a target and a range of sources.  Per source the product enters
// through the z lines, the y and x lines follow through shared memory (one copy
// of the grid, x rows padded to an odd stride), the kernel is multiplied where
// the x lines turn round, and the inverse leaves through the z lines into
// per-thread sums.  A pair costs 8 shared-memory accesses per point, four
// barriers and no global temporaries; the three-pass pipeline (split.cuh) needs
// some 20 accesses and two grids of traffic each way.  Its floor is the
// arithmetic: 6 line transforms per point, about 125 FP32 instructions at 20^3.
// Measured 13.6 thousand cycles per pair there, one CTA per SM: an HF apply of 27
// k-points (36^3, mixed) went from 4.37 to 2.03 ms, 1.81 of them here (1.77 with
// FP32 sums over all sources).
#pragma once
#include "terms.cuh"
#include "split.cuh"

namespace tcg {
namespace cube {

// twiddles by value: kernel parameters are constant-bank operands of the
// arithmetic instructions (every index is a compile-time constant)
template <typename V, int N> struct TwN {
    V w[N];
};

template <typename V, int N, int A, int B, int DIR> __device__ __forceinline__ void line(V (&x)[N], const TwN<V, N> &tw)
{
    V y[N];
#pragma unroll
    for (int t = 0; t < A; t++) {
        V u[B];
#pragma unroll
        for (int m = 0; m < B; m++) u[m] = x[t + A * m];
        sl::dft<V, B, DIR>(u);
#pragma unroll
        for (int k = 0; k < B; k++) {
            if (t * k) u[k] = DIR < 0 ? cmul(u[k], tw.w[t * k]) : cmulc(tw.w[t * k], u[k]);
            y[t + A * k] = u[k];
        }
    }
#pragma unroll
    for (int k = 0; k < B; k++) {
        V v[A];
#pragma unroll
        for (int t = 0; t < A; t++) v[t] = y[t + A * k];
        sl::dft<V, A, DIR>(v);
#pragma unroll
        for (int j = 0; j < A; j++) x[k + B * j] = v[j];
    }
}

// Sizes: the cube and, per thread, one z line and its sums in registers.
// 20^3 complex64 keeps 400 threads of about 110 registers (one CTA per SM),
// 18^3 complex128 324 of about 180; larger grids go through the passes.
// shared memory: the grid, in FP32 also its FP64 sums
template <typename T, int N> __host__ __device__ constexpr size_t cube_bytes()
{
    return (sizeof(typename C2<T>::t) * (size_t)N * N * (N + (N % 2 == 0 ? 1 : 0)) + 15) / 16 * 16;
}
template <typename T, int N> constexpr size_t smem_hf()
{
    return cube_bytes<T, N>() + (sizeof(T) == 4 ? sizeof(double2) * (size_t)N * N * N : 0);
}
template <typename T, int N> constexpr bool fits() { return sizeof(T) == 4 ? N <= 20 : N <= 18; }

template <typename T, int N>
__global__ void __launch_bounds__((N * N + 31) / 32 * 32, sl::ctas_for(N *N, sizeof(T) == 4 ? 6 * N : 9 * N))
    k_hf(CubeCall<T> a, const __grid_constant__ TwN<typename C2<T>::t, N> tw)
{
    using V = typename C2<T>::t;
    using SH = sl::ShapeOf<N>;
    constexpr int A = SH::A, B = SH::B, PX = N + (N % 2 == 0 ? 1 : 0);
    constexpr int N2 = N * N, N3 = N2 * N;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *C = reinterpret_cast<V *>(smem_raw);
    const int l = threadIdx.x;
    const bool on = l < N2;
    const int p = on ? l % N : 0, q = on ? l / N : 0;      // line: (x, y), (x, z) or (y, z)
    const int tj = blockIdx.x;
    const V *psi = a.Rpsi + (size_t)tj * N3 + (on ? l : 0);
    const int s0 = blockIdx.y * a.per, s1 = min(a.ns, s0 + a.per);
    V sum[N];
#pragma unroll
    for (int i = 0; i < N; i++) sum[i] = czero<V>();
    // FP32: the sums of every FLUSH sources are added here, each thread's to its own entries
    // (shared memory that one CTA per SM leaves free; in device memory it cost 12% of the pass)
    double2 *S = reinterpret_cast<double2 *>(smem_raw + cube_bytes<T, N>()) + (on ? l : 0);
    if (sizeof(T) == 4 && on) {
#pragma unroll
        for (int z = 0; z < N; z++) S[z * N2] = {0.0, 0.0};
    }
    V *cz = C + q * PX + p, *cy = C + q * N * PX + p, *cx = C + (q * N + p) * PX;
    for (int si = s0; si < s1; si++) {
        const V *phi = a.Rocc + (size_t)si * N3 + (on ? l : 0);
        V v[N];
        if (on) {
#pragma unroll
            for (int z = 0; z < N; z++) v[z] = cmulc(__ldg(&phi[z * N2]), __ldg(&psi[z * N2]));
            line<V, N, A, B, -1>(v, tw);
#pragma unroll
            for (int z = 0; z < N; z++) cz[z * N * PX] = v[z];
        }
        __syncthreads();
        if (on) {
#pragma unroll
            for (int y = 0; y < N; y++) v[y] = cy[y * PX];
            line<V, N, A, B, -1>(v, tw);
#pragma unroll
            for (int y = 0; y < N; y++) cy[y * PX] = v[y];
        }
        __syncthreads();
        if (on) {
            // p = y, q = z
            const T *tab = a.tab + (size_t)(a.tb[tj] * a.nSB + a.sb[si]) * N3 + q * N2 + p;
#pragma unroll
            for (int x = 0; x < N; x++) v[x] = cx[x];
            line<V, N, A, B, -1>(v, tw);
#pragma unroll
            for (int x = 0; x < N; x++) v[x] = cscale(v[x], __ldg(&tab[x * N]));
            line<V, N, A, B, +1>(v, tw);
#pragma unroll
            for (int x = 0; x < N; x++) cx[x] = v[x];
        }
        __syncthreads();
        if (on) {
#pragma unroll
            for (int y = 0; y < N; y++) v[y] = cy[y * PX];
            line<V, N, A, B, +1>(v, tw);
#pragma unroll
            for (int y = 0; y < N; y++) cy[y * PX] = v[y];
        }
        __syncthreads();
        if (on) {
            // the next source's product overwrites only the column this thread reads here
            const double f = a.fill[si];
#pragma unroll
            for (int z = 0; z < N; z++) v[z] = cz[z * N * PX];
            line<V, N, A, B, +1>(v, tw);
#pragma unroll
            for (int z = 0; z < N; z++) sum[z] = cadd(sum[z], cscale64(cmul(v[z], __ldg(&phi[z * N2])), f));
            if (sl::flush_due<V>(si - s0)) {
#pragma unroll
                for (int z = 0; z < N; z++) {
                    S[z * N2] = cadd(S[z * N2], to64(sum[z]));
                    sum[z] = czero<V>();
                }
            }
        }
    }
    if (on) {
        double2 *o = a.part + ((size_t)blockIdx.y * gridDim.x + tj) * N3 + l;
#pragma unroll
        for (int z = 0; z < N; z++) o[z * N2] = sizeof(T) == 4 ? cadd(S[z * N2], to64(sum[z])) : to64(sum[z]);
    }
}

} // namespace cube
} // namespace tcg
