// fast.cuh -- compile-time-size pass kernels for cubic grids N^3.
//
// Each 1D transform of length N is held by ONE thread in registers and run
// as a fully unrolled mixed-radix Stockham (all indices compile-time; no
// integer division, no barrier inside a line).  Shared memory only
// transposes planes between the x and y sweeps:
//   XY pass: P planes per CTA, thread (plane, line); global -> smem
//            (coalesced) -> row FFT (registers) -> smem -> column FFT
//            (registers) -> global straight from registers (coalesced: the
//            threads of a plane hold consecutive columns x).
//   Z pass : one thread per (x, y) pencil, loaded from / stored to global
//            straight from registers (consecutive threads = consecutive x);
//            the NF transformed inputs are staged in shared memory for the
//            G-space combination, each output is inverse-transformed in
//            registers and stored.
// Rows of a shared plane are padded to N+1 elements (odd stride for even N)
// so that the row sweeps are free of bank conflicts.
// Both XY passes also exist with each line split over a lane pair
// (k_xyf_pair / k_xyi_pair: N/2 values per thread, one radix-2 step through
// shuffles); each term picks one form per pass (Op::XYF_PAIR, Op::XYI_PAIR).
#pragma once
#include "fft.cuh"

namespace tcg {
namespace fast {

// ------------------------------------------------------ radix schedule --
__host__ __device__ constexpr int radix_at(int n, int s)
{
    // greedy: 8s, 4s, 2s, then odd primes; s-th radix
    int m = n, k = 0;
    while (m % 8 == 0) { if (k == s) return 8; m /= 8; k++; }
    while (m % 4 == 0) { if (k == s) return 4; m /= 4; k++; }
    while (m % 2 == 0) { if (k == s) return 2; m /= 2; k++; }
    for (int q = 3; m > 1; q += 2)
        while (m % q == 0) { if (k == s) return q; m /= q; k++; }
    return 1;
}
__host__ __device__ constexpr int nstages(int n)
{
    int s = 0;
    while (radix_at(n, s) > 1) s++;
    return s;
}
__host__ __device__ constexpr int ns_at(int n, int s)
{
    int p = 1;
    for (int i = 0; i < s; i++) p *= radix_at(n, i);
    return p;
}

template <typename V, int R, int DIR> __device__ __forceinline__ void dftR(V *v)
{
    if constexpr (R == 2) dft2<V, DIR>(v);
    else if constexpr (R == 3) dft3<V, DIR>(v);
    else if constexpr (R == 4) dft4<V, DIR>(v);
    else if constexpr (R == 5) dft5<V, DIR>(v);
    else if constexpr (R == 8) dft8<V, DIR>(v);
    else static_assert(R == 2, "unsupported radix in the fast path");
}

// one Stockham stage over a register array (Govindaraju et al. 2008 form)
template <typename V, int N, int DIR, int R, int NS>
__device__ __forceinline__ void rstage(const V (&a)[N], V (&b)[N], const V *__restrict__ tw)
{
    constexpr int M = N / R;
#pragma unroll
    for (int j = 0; j < M; j++) {
        const int k = j % NS;
        V v[R];
#pragma unroll
        for (int r = 0; r < R; r++) v[r] = a[j + r * M];
        if (NS > 1) {
#pragma unroll
            for (int r = 1; r < R; r++) {
                const int ti = k * r * (N / (NS * R));
                if (ti != 0) {
                    V w = tw[ti];
                    if (DIR > 0) w.y = -w.y;
                    v[r] = cmul(v[r], w);
                }
            }
        }
        dftR<V, R, DIR>(v);
        const int d0 = (j / NS) * NS * R + k;
#pragma unroll
        for (int r = 0; r < R; r++) b[d0 + r * NS] = v[r];
    }
}

template <typename V, int N, int DIR, int S, bool DONE = (S >= nstages(N))>
struct Stages {
    static __device__ __forceinline__ void run(V (&a)[N], V (&b)[N], const V *tw)
    {
        rstage<V, N, DIR, radix_at(N, S), ns_at(N, S)>(a, b, tw);
        Stages<V, N, DIR, S + 1>::run(b, a, tw);
    }
};
template <typename V, int N, int DIR, int S>
struct Stages<V, N, DIR, S, true> {
    static __device__ __forceinline__ void run(V (&)[N], V (&)[N], const V *) {}
};

// In-register 1D FFT of x (result in x).  tw: N twiddles exp(-2 pi i j/N).
template <typename V, int N, int DIR>
__device__ __forceinline__ void line_fft(V (&x)[N], const V *__restrict__ tw)
{
    V y[N];
    Stages<V, N, DIR, 0>::run(x, y, tw);
    if constexpr (nstages(N) % 2 == 1) {
#pragma unroll
        for (int i = 0; i < N; i++) x[i] = y[i];
    }
}

// planes per CTA (XY passes); two plane sets must fit in 227 KB of smem
template <int N, int VB> struct Cfg {
    static constexpr int P0 = (N <= 16) ? 12 : (N <= 24 ? 8 : 4);
    static constexpr int PAD = N + ((N % 2 == 0) ? 1 : 0);           // row stride in smem
    static constexpr int P = (2 * P0 * N * PAD * VB > 200 * 1024) ? P0 / 2 : P0;
    static constexpr int THREADS = P * N;
};

// asynchronous global -> shared copy of one complex element (8 or 16 B)
template <typename V>
__device__ __forceinline__ void cp_async_elem(V *dst_smem, const V *src_gmem)
{
    const unsigned d = (unsigned)__cvta_generic_to_shared(dst_smem);
    if constexpr (sizeof(V) == 16)
        asm volatile("cp.async.ca.shared.global [%0], [%1], 16;\n" ::"r"(d), "l"(src_gmem) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(d), "l"(src_gmem) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all()
{
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
}

template <typename V>
__device__ __forceinline__ void stage_tw(const GridDesc &g, V *tws, int n)
{
    const V *src = twsrc<V>(g);
    for (int i = threadIdx.x; i < n; i += blockDim.x) tws[i] = src[i];   // cubic grid: axis 0 table
}

// ---------------------------------------------------------------- XYF ----
template <typename T, int N, class Op>
__global__ void __launch_bounds__(Cfg<N, sizeof(typename C2<T>::t)>::THREADS, 3) k_xyf_fast(Op op, int nplanes)
{
    using V = typename C2<T>::t;
    constexpr int P = Cfg<N, sizeof(typename C2<T>::t)>::P, PAD = Cfg<N, sizeof(typename C2<T>::t)>::PAD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    V *A = tw + 128;
    stage_tw<V>(op.g, tw, N);
    const int pl = threadIdx.x / N, ln = threadIdx.x % N;
    const int pid0 = blockIdx.x * P;
    for (int f = 0; f < Op::NF; f++) {
        __syncthreads();
        // each thread fills column x = ln of its own plane (item and z fixed);
        // 12 elements (24 loads) in flight per thread
        if (pid0 + pl < nplanes) {
            const int item = (pid0 + pl) / N, z = (pid0 + pl) % N;
#pragma unroll 12
            for (int k = 0; k < N; k++)
                A[pl * N * PAD + k * PAD + ln] = op.xyf_load(item, f, ln, k, z, (size_t)z * N * N + (size_t)k * N + ln);
        }
        __syncthreads();
        V v[N];
        V *row = A + pl * N * PAD + ln * PAD;
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = row[i];
        line_fft<V, N, -1>(v, tw);
#pragma unroll
        for (int i = 0; i < N; i++) row[i] = v[i];
        __syncthreads();
        const V *col = A + pl * N * PAD + ln;
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = col[i * PAD];
        line_fft<V, N, -1>(v, tw);
        const int pid = pid0 + pl;
        if (pid < nplanes) {
            const int item = pid / N, z = pid % N;
            V *dst = op.tmp_grid(item, f) + (size_t)z * N * N + ln;
#pragma unroll
            for (int i = 0; i < N; i++) dst[i * N] = v[i];
        }
    }
}

// ------------------------------------------------------------------ Z ----
// Each z-line is split over a lane pair (s = lane & 1):
//   forward : one radix-2 DIF step across the pair via shuffles,
//             X[2k+s] = FFT_{N/2}( s ? (x[n] - x[n+N/2]) w^n : x[n] + x[n+N/2] )
//   inverse : FFT_{N/2} of the lane's half (frequencies 2k+s), then the
//             radix-2 DIT combine across the pair, y[n + s N/2] = E -+ w^-n O.
// Each thread holds N/2 values, so twice as many warps stay resident as
// with one thread per line.  Lanes keep the frequencies z = 2k+s for the
// G-space combination.  A CTA of 128 threads = 32 pencils x 2 halves x 2
// groups; group h handles inputs f = h, h+2, ... and outputs o = h, h+2, ...
template <typename V> __host__ __device__ constexpr int zcols() { return 32; }
constexpr int ZH = 2;

template <typename V>
__device__ __forceinline__ V shfl_xor1(V v)
{
    V r;
    r.x = __shfl_xor_sync(0xffffffffu, v.x, 1);
    r.y = __shfl_xor_sync(0xffffffffu, v.y, 1);
    return r;
}

// forward split transform: in natural order x[s*M + i] -> out X[2k+s]
template <typename V, int N>
__device__ __forceinline__ void fwd_split(V (&v)[N / 2], int s, const V *tw, const V *twM)
{
    constexpr int M = N / 2;
#pragma unroll
    for (int i = 0; i < M; i++) {
        const V o = shfl_xor1(v[i]);
        if (s == 0) v[i] = cadd(v[i], o);
        else {
            V d = csub(o, v[i]);              // x[i] - x[i+M]
            if (i != 0) d = cmul(d, tw[i]);
            v[i] = d;
        }
    }
    line_fft<V, M, -1>(v, twM);
}

// inverse split transform: in Y[2k+s] -> out natural y[s*M + n]
template <typename V, int N>
__device__ __forceinline__ void inv_split(V (&v)[N / 2], int s, const V *tw, const V *twM)
{
    constexpr int M = N / 2;
    line_fft<V, M, +1>(v, twM);               // s=0: E[n], s=1: O[n]
#pragma unroll
    for (int i = 0; i < M; i++) {
        const V o = shfl_xor1(v[i]);
        // s=0: y[n] = E + w^-n O ; s=1: y[n+M] = E - w^-n O
        V odd = s == 0 ? o : v[i];
        const V even = s == 0 ? v[i] : o;
        if (i != 0) { V w = tw[i]; w.y = -w.y; odd = cmul(odd, w); }
        v[i] = s == 0 ? cadd(even, odd) : csub(even, odd);
    }
}

template <typename T, int N, class Op>
__global__ void __launch_bounds__(128, Op::ZMINB) k_z_fast(Op op)
{
    using V = typename C2<T>::t;
    constexpr int TC = 32, M = N / 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);   // [N]: exp(-2 pi i j/N)
    V *twM = tw + 64;                          // [M]: exp(-2 pi i j/M)
    V *S = tw + 128;                           // [NF][N][TC]
    stage_tw<V>(op.g, tw, N);
    __syncthreads();
    for (int i = threadIdx.x; i < M; i += blockDim.x) twM[i] = tw[2 * i];
    __syncthreads();
    const int item = blockIdx.y;
    const int lane = threadIdx.x & 31, w = threadIdx.x >> 5;
    const int s = lane & 1;
    const int cl = (w & 1) * 16 + (lane >> 1);   // pencil within the CTA
    const int h = w >> 1;                         // group
    const int c = blockIdx.x * TC + cl;
    const bool act = c < N * N;
    const int x = op.m.tr ? c / N : c % N, y = op.m.tr ? c % N : c / N;
    V v[M];
    for (int f = h; f < Op::NF; f += ZH) {
        if (act) {
            const V *src = op.zin_grid(item, f) + c + (size_t)s * M * N * N;
#pragma unroll
            for (int i = 0; i < M; i++) v[i] = src[(size_t)i * N * N];
        } else {
#pragma unroll
            for (int i = 0; i < M; i++) v[i] = czero<V>();
        }
        fwd_split<V, N>(v, s, tw, twM);
        V *st = S + f * N * TC + cl;
#pragma unroll
        for (int k = 0; k < M; k++) st[(2 * k + s) * TC] = v[k];
    }
    __syncthreads();
    for (int o = h; o < Op::NB; o += ZH) {
#pragma unroll
        for (int k = 0; k < M; k++) {
            const int z = 2 * k + s;
            V vin[Op::NF];
#pragma unroll
            for (int f = 0; f < Op::NF; f++) vin[f] = S[f * N * TC + z * TC + cl];
            v[k] = act ? op.zmix(item, o, x, y, z, vin) : czero<V>();
        }
        if (Op::ZINV) {
            inv_split<V, N>(v, s, tw, twM);
            if (act) {
                V *dst = op.out_grid(item, o) + c + (size_t)s * M * N * N;
#pragma unroll
                for (int i = 0; i < M; i++) dst[(size_t)i * N * N] = v[i];
            }
        } else if (act) {
            // G-space output: frequencies 2k+s
            V *dst = op.out_grid(item, o) + c;
#pragma unroll
            for (int k = 0; k < M; k++) dst[(size_t)(2 * k + s) * N * N] = v[k];
        }
    }
}

// Z pass variant with one thread per z-line (ZL groups of 32 pencils split
// the inputs / outputs); used by the terms whose G-space combination is
// light (tc2x, band part of tc3a2a4b2b5), where it measured faster.
constexpr int ZL = 4;
template <typename T, int N, class Op>
__global__ void __launch_bounds__(32 * ZL, Op::ZMINB) k_z_line(Op op)
{
    using V = typename C2<T>::t;
    constexpr int TC = 32;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    V *S = tw + 128;                      // [NF][N][TC]
    stage_tw<V>(op.g, tw, N);
    __syncthreads();
    const int item = blockIdx.y;
    const int lane = threadIdx.x % TC, h = threadIdx.x / TC;
    const int c = blockIdx.x * TC + lane;
    const bool act = c < N * N;
    const int x = op.m.tr ? c / N : c % N, y = op.m.tr ? c % N : c / N;
    V v[N];
    for (int f = h; f < Op::NF; f += ZL) {
        if (act) {
            const V *src = op.zin_grid(item, f) + c;
#pragma unroll
            for (int z = 0; z < N; z++) v[z] = src[(size_t)z * N * N];
        } else {
#pragma unroll
            for (int z = 0; z < N; z++) v[z] = czero<V>();
        }
        line_fft<V, N, -1>(v, tw);
        V *st = S + f * N * TC + lane;
#pragma unroll
        for (int z = 0; z < N; z++) st[z * TC] = v[z];
    }
    __syncthreads();
    for (int o = h; o < Op::NB; o += ZL) {
#pragma unroll
        for (int z = 0; z < N; z++) {
            V vin[Op::NF];
#pragma unroll
            for (int f = 0; f < Op::NF; f++) vin[f] = S[f * N * TC + z * TC + lane];
            v[z] = act ? op.zmix(item, o, x, y, z, vin) : czero<V>();
        }
        if (Op::ZINV) line_fft<V, N, +1>(v, tw);
        if (act) {
            V *dst = op.out_grid(item, o) + c;
#pragma unroll
            for (int z = 0; z < N; z++) dst[(size_t)z * N * N] = v[z];
        }
    }
}

// ---------------------------------------------------------------- XYI ----
// smem: twiddles + GS planes-of-P (results of a group) + 1 work set
template <typename T, int N, class Op>
__global__ void __launch_bounds__(Cfg<N, sizeof(typename C2<T>::t)>::THREADS, 2) k_xyi_fast(Op op, int nplanes)
{
    using V = typename C2<T>::t;
    constexpr int P = Cfg<N, sizeof(typename C2<T>::t)>::P, PAD = Cfg<N, sizeof(typename C2<T>::t)>::PAD;
    constexpr int PS = P * N * PAD;       // one set of P planes
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    V *W = tw + 128;                      // [GS + 1][P][N][PAD]
    stage_tw<V>(op.g, tw, N);
    const int pl = threadIdx.x / N, ln = threadIdx.x % N;
    const int pid0 = blockIdx.x * P;
    const int mypid = pid0 + pl;
    const bool mine = mypid < nplanes;
    const int tj = mine ? mypid / N : 0, z = mypid % N;
    // all planes of the CTA must belong to targets with the same source count
    const int ns = op.nsrc(pid0 / N);
    // register accumulation only in the FP32 path (an FP64 column would
    // double the register footprint of the line FFT)
    constexpr bool RACC = Op::REGACC && sizeof(V) == 8;
    // BOUT: one accumulator per output grid b (GS == 1); the b loop runs
    // outside the source loop and each b's column sum is flushed on its own
    constexpr bool BOUT = RACC && Op::BOUTER;
    static_assert(!BOUT || Op::GS == 1, "per-output accumulation needs GS == 1");
    V racc[RACC ? N : 1];
    for (int bo = 0; bo < (BOUT ? Op::NB : 1); bo++) {
#pragma unroll
    for (int i = 0; i < (RACC ? N : 1); i++) racc[i] = czero<V>();
    for (int si = 0; si < ns; si++) {
        for (int b0 = BOUT ? bo : 0; b0 < (BOUT ? bo + 1 : Op::NB); b0 += Op::GS) {
            V *keepc = W + PS + pl * N * PAD + ln;      // set 1, this thread's column
#pragma unroll
            for (int q = 0; q < Op::GS; q++) {
                V *A = W;
                __syncthreads();
                // plane copies global -> smem without passing through registers
                if (mine) {   // column x = ln of this thread's own plane
                    const V *src = op.xyi_grid(op.item_of(tj, si), b0 + q) + (size_t)z * N * N + ln;
#pragma unroll
                    for (int k = 0; k < N; k++) cp_async_elem(A + pl * N * PAD + k * PAD + ln, src + (size_t)k * N);
                }
                cp_async_wait_all();
                __syncthreads();
                V v[N];
                V *row = A + pl * N * PAD + ln * PAD;
#pragma unroll
                for (int i = 0; i < N; i++) v[i] = row[i];
                line_fft<V, N, +1>(v, tw);
#pragma unroll
                for (int i = 0; i < N; i++) row[i] = v[i];
                __syncthreads();
                const V *colp = A + pl * N * PAD + ln;
#pragma unroll
                for (int i = 0; i < N; i++) v[i] = colp[i * PAD];
                line_fft<V, N, +1>(v, tw);
                if (Op::GS > 1 && q < Op::GS - 1) {
                    // keep this grid's column (thread-private) for the group accumulation
#pragma unroll
                    for (int i = 0; i < N; i++) keepc[i * PAD] = v[i];
                } else if (mine) {
                    const int item = op.item_of(tj, si);
                    if (RACC && op.regacc_grid(b0)) {
#pragma unroll
                        for (int yy = 0; yy < N; yy++) {
                            V vals[1] = {v[yy]};
                            racc[yy] = cadd(racc[yy], op.xyi_term(tj, item, b0, (size_t)z * N * N + (size_t)yy * N + ln, vals));
                            if constexpr (Op::RACC_EXTRA) op.xyi_extra(tj, item, b0, (size_t)z * N * N + (size_t)yy * N + ln, vals);
                        }
                    } else {
#pragma unroll
                        for (int yy = 0; yy < N; yy++) {
                            V vals[Op::GS];
                            if constexpr (Op::GS > 1) { vals[0] = keepc[yy * PAD]; vals[Op::GS - 1] = v[yy]; }
                            else vals[0] = v[yy];
                            op.xyi_accum(tj, item, b0, (size_t)z * N * N + (size_t)yy * N + ln, vals);
                        }
                    }
                }
                if (Op::REFWD && Op::GS == 1) {
                    // derived plane: column values -> forward column FFT -> smem -> forward rows -> global
                    const bool want = op.refwd_want(b0);
                    if (want) {
                        // per-output sums wait in this thread's own column of the
                        // read set (no other thread touches it until the next
                        // load), which frees their registers for the two FFTs
                        V *stash = A + pl * N * PAD + ln;
                        if constexpr (BOUT) {
#pragma unroll
                            for (int i = 0; i < N; i++) stash[i * PAD] = racc[i];
                        }
                        const int item = op.item_of(tj, si);
#pragma unroll
                        for (int yy = 0; yy < N; yy++)
                            v[yy] = mine ? op.refwd_load(tj, item, b0, (size_t)z * N * N + (size_t)yy * N + ln, v[yy])
                                         : czero<V>();
                        line_fft<V, N, -1>(v, tw);
                        V *B = W + PS;          // work set
                        V *cb = B + pl * N * PAD + ln;
#pragma unroll
                        for (int i = 0; i < N; i++) cb[i * PAD] = v[i];
                        __syncthreads();
                        V *rb = B + pl * N * PAD + ln * PAD;
#pragma unroll
                        for (int i = 0; i < N; i++) v[i] = rb[i];
                        line_fft<V, N, -1>(v, tw);
#pragma unroll
                        for (int i = 0; i < N; i++) rb[i] = v[i];
                        __syncthreads();
                        if (mine) {
                            V *dstp = op.refwd_grid(op.item_of(tj, si), b0) + (size_t)z * N * N + ln;
#pragma unroll 4
                            for (int k = 0; k < N; k++) dstp[(size_t)k * N] = B[pl * N * PAD + k * PAD + ln];
                        }
                        if constexpr (BOUT) {
#pragma unroll
                            for (int i = 0; i < N; i++) racc[i] = stash[i * PAD];
                        }
                    }
                }
            }
        }
    }
    if constexpr (BOUT) {
        if (mine && op.regacc_grid(bo)) {
#pragma unroll
            for (int yy = 0; yy < N; yy++) op.xyi_flush_b(tj, bo, (size_t)z * N * N + (size_t)yy * N + ln, racc[yy]);
        }
    }
    }
    if (RACC && !BOUT && mine) {
#pragma unroll
        for (int yy = 0; yy < N; yy++) op.xyi_flush(tj, (size_t)z * N * N + (size_t)yy * N + ln, racc[yy]);
    }
}

// XYI with the next plane set prefetched: for terms without re-forwarded or
// grouped grids (GS == 1, no REFWD) the two plane sets alternate, and the
// asynchronous copies of step it + 1 (source, output grid) are in flight
// while step it is transformed and accumulated.
template <typename T, int N, class Op>
__global__ void __launch_bounds__(Cfg<N, sizeof(typename C2<T>::t)>::THREADS, 2) k_xyi_pf(Op op, int nplanes)
{
    using V = typename C2<T>::t;
    static_assert(Op::GS == 1, "prefetching XYI handles ungrouped outputs only");
    constexpr int P = Cfg<N, sizeof(V)>::P, PAD = Cfg<N, sizeof(V)>::PAD;
    constexpr int PS = P * N * PAD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    V *W = tw + 128;                      // [2][P][N][PAD], alternating
    stage_tw<V>(op.g, tw, N);
    const int pl = threadIdx.x / N, ln = threadIdx.x % N;
    const int pid0 = blockIdx.x * P;
    const int mypid = pid0 + pl;
    const bool mine = mypid < nplanes;
    const int tj = mine ? mypid / N : 0, z = mypid % N;
    const int ns = op.nsrc(pid0 / N);
    constexpr bool RACC = Op::REGACC && sizeof(V) == 8;
    static_assert(!(RACC && Op::REFWD), "re-forwarded outputs accumulate through xyi_accum");
    V racc[RACC ? N : 1];
#pragma unroll
    for (int i = 0; i < (RACC ? N : 1); i++) racc[i] = czero<V>();
    const int total = ns * Op::NB;        // steps: it = si * NB + b
    auto issue = [&](int it) {
        if (mine) {
            const V *src = op.xyi_grid(op.item_of(tj, it / Op::NB), it % Op::NB) + (size_t)z * N * N + ln;
            V *dst = W + (it & 1) * PS + pl * N * PAD + ln;
#pragma unroll
            for (int k = 0; k < N; k++) cp_async_elem(dst + k * PAD, src + (size_t)k * N);
        }
        asm volatile("cp.async.commit_group;\n" ::: "memory");
    };
    issue(0);
    for (int it = 0; it < total; it++) {
        __syncthreads();                  // every thread is done with the set that step it + 1 overwrites
        if (it + 1 < total) {
            issue(it + 1);
            asm volatile("cp.async.wait_group 1;\n" ::: "memory");
        } else {
            asm volatile("cp.async.wait_group 0;\n" ::: "memory");
        }
        __syncthreads();
        const int si = it / Op::NB, b0 = it % Op::NB;
        V *A = W + (it & 1) * PS;
        V v[N];
        V *row = A + pl * N * PAD + ln * PAD;
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = row[i];
        line_fft<V, N, +1>(v, tw);
#pragma unroll
        for (int i = 0; i < N; i++) row[i] = v[i];
        __syncthreads();
        const V *colp = A + pl * N * PAD + ln;
#pragma unroll
        for (int i = 0; i < N; i++) v[i] = colp[i * PAD];
        line_fft<V, N, +1>(v, tw);
        if (mine) {
            const int item = op.item_of(tj, si);
            if (RACC && op.regacc_grid(b0)) {
#pragma unroll
                for (int yy = 0; yy < N; yy++) {
                    V vals[1] = {v[yy]};
                    racc[yy] = cadd(racc[yy], op.xyi_term(tj, item, b0, (size_t)z * N * N + (size_t)yy * N + ln, vals));
                    if constexpr (Op::RACC_EXTRA) op.xyi_extra(tj, item, b0, (size_t)z * N * N + (size_t)yy * N + ln, vals);
                }
            } else {
#pragma unroll
                for (int yy = 0; yy < N; yy++) {
                    V vals[1] = {v[yy]};
                    op.xyi_accum(tj, item, b0, (size_t)z * N * N + (size_t)yy * N + ln, vals);
                }
            }
        }
        if (Op::REFWD && op.refwd_want(b0)) {   // uniform over the CTA
            // derived plane, transformed forward in place in the current set:
            // columns (registers) -> own column -> rows -> global
            __syncthreads();                      // every column of the set has been read
            const int item = op.item_of(tj, si);
#pragma unroll
            for (int yy = 0; yy < N; yy++)
                v[yy] = mine ? op.refwd_load(tj, item, b0, (size_t)z * N * N + (size_t)yy * N + ln, v[yy]) : czero<V>();
            line_fft<V, N, -1>(v, tw);
            V *cb = A + pl * N * PAD + ln;
#pragma unroll
            for (int i = 0; i < N; i++) cb[i * PAD] = v[i];
            __syncthreads();
#pragma unroll
            for (int i = 0; i < N; i++) v[i] = row[i];
            line_fft<V, N, -1>(v, tw);
#pragma unroll
            for (int i = 0; i < N; i++) row[i] = v[i];
            __syncthreads();
            if (mine) {
                V *dstp = op.refwd_grid(item, b0) + (size_t)z * N * N + ln;
#pragma unroll 4
                for (int k = 0; k < N; k++) dstp[(size_t)k * N] = A[pl * N * PAD + k * PAD + ln];
            }
        }
    }
    if (RACC && mine) {
#pragma unroll
        for (int yy = 0; yy < N; yy++) op.xyi_flush(tj, (size_t)z * N * N + (size_t)yy * N + ln, racc[yy]);
    }
}

// ------------------------------------------------- XY passes, line pairs --
// The same XY passes with each row / column split over a lane pair
// (s = lane & 1, as in the Z pass): half the registers per thread, so twice
// the warps stay resident.  Forward lines: natural halves x = s M + i in,
// frequencies 2k + s out (fwd_split); inverse lines: frequencies 2k + s in,
// natural halves out (inv_split).  Pairs are adjacent lanes, so a CTA holds
// whole warps: P N is a multiple of 16.
__host__ __device__ constexpr int gcd_c(int a, int b) { return b == 0 ? a : gcd_c(b, a % b); }
template <int N, int VB> struct CfgP {
    static constexpr int Q = 16 / gcd_c(N, 16);
    static constexpr int P = (96 + Q * N - 1) / (Q * N) * Q;         // >= 96 lines per CTA
    static constexpr int PAD = N + ((N % 2 == 0) ? 1 : 0);
    static constexpr int THREADS = 2 * P * N;
    // register cap: FP32 keeps >= 16 warps per SM, FP64 one CTA's worth
    static constexpr int CTAS = VB == 8 ? (512 + THREADS - 1) / THREADS : 1;
    static constexpr int REG0 = (65536 / (CTAS * THREADS)) & ~7;
    static constexpr int REG = REG0 < 168 ? REG0 : 168;
    static_assert(THREADS % 32 == 0, "line pairs need whole warps");
};

template <typename T, int N, class Op>
__global__ void __launch_bounds__(CfgP<N, sizeof(typename C2<T>::t)>::THREADS)
    __maxnreg__((CfgP<N, sizeof(typename C2<T>::t)>::REG)) k_xyf_pair(Op op, int nplanes)
{
    using V = typename C2<T>::t;
    using CF = CfgP<N, sizeof(V)>;
    constexpr int P = CF::P, PAD = CF::PAD, M = N / 2;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);   // [N]
    V *twM = tw + 64;                          // [M]
    V *A = tw + 128;
    stage_tw<V>(op.g, tw, N);
    __syncthreads();
    for (int i = threadIdx.x; i < M; i += blockDim.x) twM[i] = tw[2 * i];
    const int s = threadIdx.x & 1, pi = threadIdx.x >> 1;
    const int pl = pi / N, ln = pi % N;
    const int pid0 = blockIdx.x * P;
    for (int f = 0; f < Op::NF; f++) {
        __syncthreads();
        // the 2N threads of a plane fill it: element r0 + 2 k N, r0 = 2 ln + s
        if (pid0 + pl < nplanes) {
            const int item = (pid0 + pl) / N, z = (pid0 + pl) % N;
            const int r0 = 2 * ln + s, x0 = r0 % N, y0 = r0 / N;
#pragma unroll 6
            for (int k = 0; k < M; k++) {
                const int y = y0 + 2 * k;
                A[pl * N * PAD + y * PAD + x0] = op.xyf_load(item, f, x0, y, z, (size_t)z * N * N + (size_t)y * N + x0);
            }
        }
        __syncthreads();
        V v[M];
        V *row = A + pl * N * PAD + ln * PAD;
#pragma unroll
        for (int i = 0; i < M; i++) v[i] = row[s * M + i];
        fwd_split<V, N>(v, s, tw, twM);
        __syncwarp();
#pragma unroll
        for (int k = 0; k < M; k++) row[2 * k + s] = v[k];
        __syncthreads();
        const V *col = A + pl * N * PAD + ln;
#pragma unroll
        for (int i = 0; i < M; i++) v[i] = col[(s * M + i) * PAD];
        fwd_split<V, N>(v, s, tw, twM);
        const int pid = pid0 + pl;
        if (pid < nplanes) {
            const int item = pid / N, z = pid % N;
            V *dst = op.tmp_grid(item, f) + (size_t)z * N * N + ln;
#pragma unroll
            for (int k = 0; k < M; k++) dst[(2 * k + s) * N] = v[k];
        }
    }
}

template <typename T, int N, class Op>
__global__ void __launch_bounds__(CfgP<N, sizeof(typename C2<T>::t)>::THREADS)
    __maxnreg__((CfgP<N, sizeof(typename C2<T>::t)>::REG)) k_xyi_pair(Op op, int nplanes)
{
    using V = typename C2<T>::t;
    using CF = CfgP<N, sizeof(V)>;
    constexpr int P = CF::P, PAD = CF::PAD, M = N / 2;
    constexpr int PS = P * N * PAD;       // one set of P planes
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *tw = reinterpret_cast<V *>(smem_raw);
    V *twM = tw + 64;
    V *W = tw + 128;                      // [2][P][N][PAD]: read set, keep / work set
    stage_tw<V>(op.g, tw, N);
    __syncthreads();
    for (int i = threadIdx.x; i < M; i += blockDim.x) twM[i] = tw[2 * i];
    const int s = threadIdx.x & 1, pi = threadIdx.x >> 1;
    const int pl = pi / N, ln = pi % N;
    const int pid0 = blockIdx.x * P;
    const int mypid = pid0 + pl;
    const bool mine = mypid < nplanes;
    const int tj = mine ? mypid / N : 0, z = mypid % N;
    // all planes of the CTA must belong to targets with the same source count
    const int ns = op.nsrc(pid0 / N);
    constexpr bool RACC = Op::REGACC && sizeof(V) == 8;
    constexpr bool BOUT = RACC && Op::BOUTER;
    static_assert(!BOUT || Op::GS == 1, "per-output accumulation needs GS == 1");
    // this thread's rows y = s M + n of its column, as element offsets
    const size_t pz = (size_t)z * N * N + ln + (size_t)s * M * N;
    // plane copies: this thread moves elements r0 + 2 k N of its own plane
    const int r0 = 2 * ln + s, x0 = r0 % N, y0 = r0 / N;
    V racc[RACC ? M : 1];
    for (int bo = 0; bo < (BOUT ? Op::NB : 1); bo++) {
#pragma unroll
        for (int i = 0; i < (RACC ? M : 1); i++) racc[i] = czero<V>();
        for (int si = 0; si < ns; si++) {
            for (int b0 = BOUT ? bo : 0; b0 < (BOUT ? bo + 1 : Op::NB); b0 += Op::GS) {
                V *keepc = W + PS + pl * N * PAD + ln + s * M * PAD;   // set 1: this thread's half column
#pragma unroll
                for (int q = 0; q < Op::GS; q++) {
                    V *A = W;
                    __syncthreads();
                    if (mine) {   // element r0 + 2 k N of this thread's own plane
                        const V *src = op.xyi_grid(op.item_of(tj, si), b0 + q) + (size_t)z * N * N + (size_t)y0 * N + x0;
                        V *dsm = A + pl * N * PAD + y0 * PAD + x0;
#pragma unroll
                        for (int k = 0; k < M; k++) cp_async_elem(dsm + 2 * k * PAD, src + (size_t)2 * k * N);
                    }
                    cp_async_wait_all();
                    __syncthreads();
                    V v[M];
                    V *row = A + pl * N * PAD + ln * PAD;
#pragma unroll
                    for (int k = 0; k < M; k++) v[k] = row[2 * k + s];
                    inv_split<V, N>(v, s, tw, twM);
                    __syncwarp();
#pragma unroll
                    for (int i = 0; i < M; i++) row[s * M + i] = v[i];
                    __syncthreads();
                    V *colp = A + pl * N * PAD + ln;
#pragma unroll
                    for (int k = 0; k < M; k++) v[k] = colp[(2 * k + s) * PAD];
                    inv_split<V, N>(v, s, tw, twM);            // v[n]: row y = s M + n
                    if (Op::GS > 1 && q < Op::GS - 1) {
#pragma unroll
                        for (int i = 0; i < M; i++) keepc[i * PAD] = v[i];
                    } else if (mine) {
                        const int item = op.item_of(tj, si);
                        if (RACC && op.regacc_grid(b0)) {
#pragma unroll
                            for (int i = 0; i < M; i++) {
                                V vals[1] = {v[i]};
                                racc[i] = cadd(racc[i], op.xyi_term(tj, item, b0, pz + (size_t)i * N, vals));
                                if constexpr (Op::RACC_EXTRA) op.xyi_extra(tj, item, b0, pz + (size_t)i * N, vals);
                            }
                        } else {
#pragma unroll
                            for (int i = 0; i < M; i++) {
                                V vals[Op::GS];
                                if constexpr (Op::GS > 1) { vals[0] = keepc[i * PAD]; vals[Op::GS - 1] = v[i]; }
                                else vals[0] = v[i];
                                op.xyi_accum(tj, item, b0, pz + (size_t)i * N, vals);
                            }
                        }
                    }
                    if (Op::REFWD && Op::GS == 1) {
                        const bool want = op.refwd_want(b0);   // uniform over the CTA
                        if (want) {
                            // the column sums wait in the slots this thread read
                            V *stash = colp + s * PAD;
                            if constexpr (BOUT) {
#pragma unroll
                                for (int k = 0; k < M; k++) stash[2 * k * PAD] = racc[k];
                            }
                            const int item = op.item_of(tj, si);
#pragma unroll
                            for (int i = 0; i < M; i++)
                                v[i] = mine ? op.refwd_load(tj, item, b0, pz + (size_t)i * N, v[i]) : czero<V>();
                            fwd_split<V, N>(v, s, tw, twM);          // frequencies y = 2k + s
                            V *B = W + PS;
                            V *cb = B + pl * N * PAD + ln;
#pragma unroll
                            for (int k = 0; k < M; k++) cb[(2 * k + s) * PAD] = v[k];
                            __syncthreads();
                            V *rb = B + pl * N * PAD + ln * PAD;
#pragma unroll
                            for (int i = 0; i < M; i++) v[i] = rb[s * M + i];
                            fwd_split<V, N>(v, s, tw, twM);
                            __syncwarp();
#pragma unroll
                            for (int k = 0; k < M; k++) rb[2 * k + s] = v[k];
                            __syncthreads();
                            if (mine) {
                                V *dstp = op.refwd_grid(op.item_of(tj, si), b0) + (size_t)z * N * N + (size_t)y0 * N + x0;
                                const V *bs = B + pl * N * PAD + y0 * PAD + x0;
#pragma unroll 6
                                for (int k = 0; k < M; k++) dstp[(size_t)2 * k * N] = bs[2 * k * PAD];
                            }
                            if constexpr (BOUT) {
#pragma unroll
                                for (int k = 0; k < M; k++) racc[k] = stash[2 * k * PAD];
                            }
                        }
                    }
                }
            }
        }
        if constexpr (BOUT) {
            if (mine && op.regacc_grid(bo)) {
#pragma unroll
                for (int i = 0; i < M; i++) op.xyi_flush_b(tj, bo, pz + (size_t)i * N, racc[i]);
            }
        }
    }
    if (RACC && !BOUT && mine) {
#pragma unroll
        for (int i = 0; i < M; i++) op.xyi_flush(tj, pz + (size_t)i * N, racc[i]);
    }
}

template <typename V, int N> __host__ inline size_t smem_xy_pair(int sets)
{
    return sizeof(V) * (128 + (size_t)sets * CfgP<N, sizeof(V)>::P * N * CfgP<N, sizeof(V)>::PAD);
}

template <typename V, int N> __host__ inline size_t smem_xy_fast(int sets)
{
    return sizeof(V) * (128 + (size_t)sets * Cfg<N, sizeof(V)>::P * N * Cfg<N, sizeof(V)>::PAD);
}
template <typename V, int N> __host__ inline size_t smem_z_fast(int nf)
{
    return sizeof(V) * (128 + (size_t)nf * N * zcols<V>());
}

} // namespace fast
} // namespace tcg
