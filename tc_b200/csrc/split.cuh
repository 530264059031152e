// split.cuh -- pass kernels for cubic grids N^3 that transform each line in
// registers of several threads.
//
// N = A * B (A >= B).  A line is transformed by the two-step algorithm of
// Cooley and Tukey (n = t + p m, k = k1 + q k2 with {p, q} = {A, B}):
//   step 1, thread t < p: u_t[k1] = w_N^{t k1} DFT_q over m of x[t + p m];
//   step 2, thread t < q (k1 = t): X[t + q k2] = DFT_p over t' of u_t'[k1],
// with one exchange through shared memory between the steps and registers at
// both ends.  Forward transforms take (p, q) = (A, B), inverse ones (B, A), so
// that a forward transform may start from the registers an inverse one ended
// with, and the reverse.
//
// In a z-plane the real-space side is stored x fastest and the G side y
// fastest: the XY passes read and write both straight between global memory
// and registers, with consecutive threads on consecutive elements, and need
// three exchanges per two-dimensional transform (inside the first line
// transform, between the two, inside the second).  Two buffers take turns,
// so each exchange costs one barrier: the buffer written after a barrier was
// last read before it.
//
// What bounds these kernels is the shared-memory pipe: 6 accesses per element
// of a 2-D transform (a whole line per thread needs 4 but holds N values per
// thread, which leaves a third of the warps resident; the earlier split
// form, which staged planes in shared memory, made 8 to 10 with 3 times the
// barriers).
#pragma once
#include <type_traits>
#include "fft.cuh"
#include "fast.cuh"

namespace tcg {
namespace sl {

template <int N_, int A_, int B_> struct Shape {
    static constexpr int N = N_, A = A_, B = B_;
    static constexpr int PAD = N_ + ((N_ % 2 == 0) ? 1 : 0);   // odd row stride: rows across lanes conflict-free
    // XY passes: one plane per CTA, A groups of LP lanes.  A group of N lanes
    // that ends inside a half-warp would share its shared-memory accesses with the
    // next group's row, two to a bank (30: every second access took a third
    // wavefront), so it is padded to a half-warp or warp where that is close.
    static constexpr int LP = N_ <= 16 ? 16 : (N_ <= 32 ? 32 : N_);
    static constexpr int THREADS = A_ * LP;
    static constexpr int ZTHREADS = A_ * 32;     // Z pass: 32 pencils per CTA
    static_assert(N_ == A_ * B_ && A_ >= B_ && N_ <= 64, "two-step lines; pencil masks hold 64 bits");
};
// compiled sizes; near-square factors keep both steps' threads busy
template <int N> struct ShapeOf { static constexpr int A = 0, B = 0; };
template <> struct ShapeOf<12> { static constexpr int A = 4, B = 3; };
template <> struct ShapeOf<15> { static constexpr int A = 5, B = 3; };
template <> struct ShapeOf<16> { static constexpr int A = 4, B = 4; };
template <> struct ShapeOf<18> { static constexpr int A = 6, B = 3; };
template <> struct ShapeOf<20> { static constexpr int A = 5, B = 4; };
template <> struct ShapeOf<24> { static constexpr int A = 6, B = 4; };
template <> struct ShapeOf<25> { static constexpr int A = 5, B = 5; };
template <> struct ShapeOf<27> { static constexpr int A = 9, B = 3; };
template <> struct ShapeOf<30> { static constexpr int A = 6, B = 5; };
template <> struct ShapeOf<32> { static constexpr int A = 8, B = 4; };
template <> struct ShapeOf<36> { static constexpr int A = 6, B = 6; };
template <> struct ShapeOf<40> { static constexpr int A = 8, B = 5; };
template <> struct ShapeOf<45> { static constexpr int A = 9, B = 5; };
template <> struct ShapeOf<48> { static constexpr int A = 8, B = 6; };

// resident CTAs per SM that leave `regs` registers per thread
__host__ __device__ constexpr int ctas_for(int threads, int regs)
{
    const int w = (threads + 31) / 32 * 32;
    int c = 65536 / (w * regs);
    if (c * w > 2048) c = 2048 / w;
    return c < 1 ? 1 : c;
}

// ------------------------------------------------------- short DFTs --------
// 6 = 2 x 3 by the prime-factor map (Good 1958: no twiddles); 9 = 3 x 3
template <typename V, int DIR> __device__ __forceinline__ void dft6(V *v)
{
    V a[3] = {v[0], v[2], v[4]}, b[3] = {v[3], v[5], v[1]};
    dft3<V, DIR>(a);
    dft3<V, DIR>(b);
    v[0] = cadd(a[0], b[0]);
    v[3] = csub(a[0], b[0]);
    v[4] = cadd(a[1], b[1]);
    v[1] = csub(a[1], b[1]);
    v[2] = cadd(a[2], b[2]);
    v[5] = csub(a[2], b[2]);
}
template <typename V, int DIR> __device__ __forceinline__ void dft9(V *v)
{
    using S = decltype(v[0].x);
    // cos, sin of 2 pi j / 9, j = 1, 2, 4
    const S c1 = (S)0.76604444311897803520, s1 = (S)0.64278760968653932632;
    const S c2 = (S)0.17364817766693034885, s2 = (S)0.98480775301220805937;
    const S c4 = (S)-0.93969262078590838405, s4 = (S)0.34202014332566873304;
    auto rot = [](V a, S c, S s) { return V{a.x * c - (S)DIR * a.y * s, a.y * c + (S)DIR * a.x * s}; };
    V a[3] = {v[0], v[3], v[6]}, b[3] = {v[1], v[4], v[7]}, d[3] = {v[2], v[5], v[8]};
    dft3<V, DIR>(a);
    dft3<V, DIR>(b);
    dft3<V, DIR>(d);
    b[1] = rot(b[1], c1, s1);
    b[2] = rot(b[2], c2, s2);
    d[1] = rot(d[1], c2, s2);
    d[2] = rot(d[2], c4, s4);
#pragma unroll
    for (int k = 0; k < 3; k++) {
        V w[3] = {a[k], b[k], d[k]};
        dft3<V, DIR>(w);
        v[k] = w[0];
        v[k + 3] = w[1];
        v[k + 6] = w[2];
    }
}
template <typename V, int DIR> __device__ __forceinline__ void dft7(V *v)
{
    using S = decltype(v[0].x);
    // cos, sin of 2 pi j / 7
    constexpr double c[4] = {1.0, 0.62348980185873353053, -0.22252093395631440429, -0.90096886790241912624};
    constexpr double w[4] = {0.0, 0.78183148246802980871, 0.97492791218182360702, 0.43388373911755812048};
    V t[4], d[4], a = v[0];
#pragma unroll
    for (int k = 1; k < 4; k++) {
        t[k] = cadd(v[k], v[7 - k]);
        d[k] = csub(v[k], v[7 - k]);
    }
    v[0] = cadd(cadd(a, t[1]), cadd(t[2], t[3]));
    auto sum3 = [](S x, double p, S y, double q, S z, double r) { return CMul::mul2(x, p, y, q) + CMul::mul(z, r); };
#pragma unroll
    for (int j = 1; j < 4; j++) {
        // j k mod 7 folded to 1..3; the sine changes sign beyond
        const int i1 = j, i2 = 2 * j % 7 > 3 ? 7 - 2 * j % 7 : 2 * j % 7, i3 = 3 * j % 7 > 3 ? 7 - 3 * j % 7 : 3 * j % 7;
        const double g2 = 2 * j % 7 > 3 ? -1.0 : 1.0, g3 = 3 * j % 7 > 3 ? -1.0 : 1.0;
        const V m = {a.x + sum3(t[1].x, c[i1], t[2].x, c[i2], t[3].x, c[i3]),
                     a.y + sum3(t[1].y, c[i1], t[2].y, c[i2], t[3].y, c[i3])};
        const V n = cmuli(V{sum3(d[1].x, w[i1], d[2].x, g2 * w[i2], d[3].x, g3 * w[i3]),
                            sum3(d[1].y, w[i1], d[2].y, g2 * w[i2], d[3].y, g3 * w[i3])}, DIR);
        v[j] = cadd(m, n);
        v[7 - j] = csub(m, n);
    }
}
template <typename V, int R, int DIR> __device__ __forceinline__ void dft(V *v)
{
    if constexpr (R == 6) dft6<V, DIR>(v);
    else if constexpr (R == 7) dft7<V, DIR>(v);
    else if constexpr (R == 9) dft9<V, DIR>(v);
    else fast::dftR<V, R, DIR>(v);
}

// step-1 factors w_N^{t k1}, k1 = 1 .. Q - 1, of a thread (forward sign)
template <typename V, int Q> struct Tw {
    V w[Q];
    __device__ __forceinline__ void load(const GridDesc &g, int t)
    {
        const V *src = twsrc<V>(g);
#pragma unroll
        for (int k = 1; k < Q; k++) w[k] = __ldg(&src[t * k]);
    }
    __device__ __forceinline__ V operator()(int k) const { return w[k]; }
};
// the same read from a table in shared memory when needed
template <typename V> struct TwS {
    const V *tab;
    int t;
    __device__ __forceinline__ V operator()(int k) const { return tab[t * k]; }
};
template <typename V, int Q, int DIR, class TW> __device__ __forceinline__ void step1(V (&u)[Q], const TW &tw)
{
    dft<V, Q, DIR>(u);
#pragma unroll
    for (int k = 1; k < Q; k++) {
        const V w = tw(k);
        u[k] = DIR < 0 ? cmul(u[k], w) : cmulc(w, u[k]);
    }
}
// exchange: u[k1] of thread t goes to buf[(k1 P + t) stride], thread t < Q reads its P values
template <typename V, int P, int Q> __device__ __forceinline__ void put(V *buf, int stride, int t, const V (&u)[Q])
{
#pragma unroll
    for (int k = 0; k < Q; k++) buf[(k * P + t) * stride] = u[k];
}
template <typename V, int P, int Q, int DIR> __device__ __forceinline__ void step2(const V *buf, int stride, int t, V (&v)[P])
{
#pragma unroll
    for (int j = 0; j < P; j++) v[j] = buf[(t * P + j) * stride];
    dft<V, P, DIR>(v);
}

// Forward XY transform of one plane.  In: u[m] = f(x = l, y = t + A m), t < A.
// Out: v[m] = F(kx = t + B m, ky = l), t < B.  b0, b1: the two buffers; b0 holds
// the last exchange, so the caller swaps them for its next transform.
template <typename V, class S, class TW>
__device__ __forceinline__ void plane_fwd(V *b0, V *b1, int t, int l, V (&u)[S::B], const TW &tw, V (&v)[S::A])
{
    constexpr int A = S::A, B = S::B, PAD = S::PAD;
    const bool on = S::LP == S::N || l < S::N;
    if (on) {
        step1<V, B, -1>(u, tw);
        put<V, A, B>(b0 + l, PAD, t, u);
    }
    __syncthreads();
    if (on && t < B) {
        step2<V, A, B, -1>(b0 + l, PAD, t, v);          // ky = t + B m at x = l
#pragma unroll
        for (int m = 0; m < A; m++) b1[(t + B * m) * PAD + l] = v[m];
    }
    __syncthreads();
    if (on) {
#pragma unroll
        for (int m = 0; m < B; m++) u[m] = b1[l * PAD + t + A * m];   // x = t + A m at ky = l
        step1<V, B, -1>(u, tw);
        put<V, A, B>(b0 + l, PAD, t, u);
    }
    __syncthreads();
    if (on && t < B) step2<V, A, B, -1>(b0 + l, PAD, t, v);
}
// Inverse XY transform.  In: u[m] = F(kx = t + B m, ky = l), t < B.
// Out: v[m] = f(x = l, y = t + A m), t < A.
template <typename V, class S, class TW>
__device__ __forceinline__ void plane_inv(V *b0, V *b1, int t, int l, V (&u)[S::A], const TW &tw, V (&v)[S::B])
{
    constexpr int A = S::A, B = S::B, PAD = S::PAD;
    const bool on = S::LP == S::N || l < S::N;
    if (on && t < B) {
        step1<V, A, +1>(u, tw);
        put<V, B, A>(b0 + l, PAD, t, u);
    }
    __syncthreads();
    if (on) {
        step2<V, B, A, +1>(b0 + l, PAD, t, v);          // x = t + A m at ky = l
#pragma unroll
        for (int m = 0; m < B; m++) b1[l * PAD + t + A * m] = v[m];
    }
    __syncthreads();
    if (on && t < B) {
#pragma unroll
        for (int m = 0; m < A; m++) u[m] = b1[(t + B * m) * PAD + l];   // ky = t + B m at x = l
        step1<V, A, +1>(u, tw);
        put<V, B, A>(b0 + l, PAD, t, u);
    }
    __syncthreads();
    if (on) step2<V, B, A, +1>(b0 + l, PAD, t, v);
}

// --------------------------------------------------------------- XYF --------
// One (item, z) plane per CTA: pair products -> forward XY -> tmp (y fastest).
// For ops without a target / source structure (Op::NSO == 0).
template <typename T, class Op, class S>
__global__ void __launch_bounds__(S::THREADS, ctas_for(S::THREADS, sizeof(T) == 4 ? 56 : 104)) k_xyf_items(Op op, int items)
{
    using V = typename C2<T>::t;
    constexpr int N = S::N, A = S::A, B = S::B, PS = S::N * S::PAD;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *b0 = reinterpret_cast<V *>(smem_raw), *b1 = b0 + PS;
    const int t = threadIdx.x / S::LP, l = threadIdx.x % S::LP;
    const bool on = S::LP == N || l < N;
    const int z = blockIdx.x / items, item = blockIdx.x % items;
    const size_t pz = (size_t)z * N * N;
    Tw<V, B> tw;
    tw.load(op.g, t);
    for (int f = 0; f < Op::NF; f++) {
        V u[B], v[A];
        if (on) {
#pragma unroll
            for (int m = 0; m < B; m++) {
                const int y = t + A * m;
                u[m] = op.xyf_load(item, f, l, y, z, pz + (size_t)y * N + l);
            }
        }
        plane_fwd<V, S>(b0, b1, t, l, u, tw, v);
        if (on && t < B) {
            V *dst = op.tmp_grid(item, f) + pz + l;
#pragma unroll
            for (int m = 0; m < A; m++) dst[(size_t)(t + B * m) * N] = v[m];
        }
        V *s = b0;
        b0 = b1;
        b1 = s;
    }
}

__device__ __forceinline__ void cp_commit() { asm volatile("cp.async.commit_group;\n" ::: "memory"); }
template <int K> __device__ __forceinline__ void cp_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(K) : "memory"); }

// One (target, z) plane per CTA, looping over `per` of the chunk's sources (part
// blockIdx.y): the target's operand planes are read again for every source from
// L1, the source's own (at most Op::NSO per input) are copied ahead, one input
// while the previous one is transformed, into slots that belong to the reading
// thread.  With a CTA per pair every operand came from L2 for every pair (3bX:xyf
// at 30^3: 7 TB/s of it).
template <typename T, class Op, class S>
__global__ void __launch_bounds__(S::THREADS, ctas_for(S::THREADS, sizeof(T) == 4 ? 64 : 104)) k_xyf(Op op, int nt, int per)
{
    using V = typename C2<T>::t;
    constexpr int N = S::N, A = S::A, B = S::B, PS = S::N * S::PAD, NO = Op::NSO;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *b0 = reinterpret_cast<V *>(smem_raw), *b1 = b0 + PS;
    V *ops = b1 + PS + threadIdx.x;              // [NO][B][THREADS]
    const int t = threadIdx.x / S::LP, l = threadIdx.x % S::LP;
    const bool on = S::LP == N || l < N;
    const int z = blockIdx.x / nt, tj = blockIdx.x % nt;
    const size_t pz = (size_t)z * N * N, p0 = pz + (size_t)t * N + l;
    const int s0 = blockIdx.y * per, s1 = min(op.nsrc(tj), s0 + per);
    Tw<V, B> tw;
    tw.load(op.g, t);
    auto fetch = [&](int si, int f) {
        if (on) {
#pragma unroll
            for (int k = 0; k < NO; k++) {
                const V *src = op.xyf_operand(k, f, si);
                if (src) {
#pragma unroll
                    for (int m = 0; m < B; m++) fast::cp_async_elem(ops + (k * B + m) * S::THREADS, src + p0 + (size_t)A * m * N);
                }
            }
        }
        cp_commit();
    };
    fetch(s0, 0);
#pragma unroll 1
    for (int si = s0; si < s1; si++) {
        const int item = op.item_of(tj, si);
        unsigned long long bits = ~0ull;
        if (Op::BLI != 0 && op.m.prune && on) bits = op.pcol(item, l);   // kx mask of row ky = l
        bits >>= t;
#pragma unroll 1
        for (int f = 0; f < Op::NF; f++) {
            V u[B], v[A];
            cp_wait<0>();
            if (on) {
#pragma unroll
                for (int m = 0; m < B; m++) {
                    V o[NO];
#pragma unroll
                    for (int k = 0; k < NO; k++) o[k] = ops[(k * B + m) * S::THREADS];
                    u[m] = op.xyf_pair(tj, f, p0 + (size_t)A * m * N, o);
                }
            }
            if (f + 1 < Op::NF) fetch(si, f + 1);
            else if (si + 1 < s1) fetch(si + 1, 0);
            plane_fwd<V, S>(b0, b1, t, l, u, tw, v);
            if (on && t < B) {
                V *dst = op.tmp_grid(item, f) + pz + (size_t)t * N + l;
                const bool bl = (Op::BLI >> f) & 1;
#pragma unroll
                for (int m = 0; m < A; m++)
                    if (!bl || ((bits >> (B * m)) & 1)) dst[(size_t)B * m * N] = v[m];
            }
            V *s = b0;
            b0 = b1;
            b1 = s;
        }
    }
}
template <typename V, class S, class Op> __host__ inline size_t smem_xyf()
{
    return sizeof(V) * (2 * (size_t)S::N * S::PAD + (size_t)Op::NSO * S::B * S::THREADS);
}

// --------------------------------------------------------------- XYI --------
// One (target, z) plane per CTA.  The outputs b (in groups of GS) run outside,
// the chunk's sources inside, and a group's sums over the sources (at most
// Op::NACC of them: xyi_add) stay with the thread that owns the points, in
// registers; each reaches the FP64 accumulators once per group and chunk, in FP32
// after every FLUSH sources (xyi_put).
// What bounds the pass is the latency of its operands (phi_q, grad phi_q, Q_q at
// the plane: read by every target, so from L2): loaded where they are used, they
// stalled each step for longer than its transforms took (issue slots 27% busy,
// 10.7 of 14 stall cycles long_scoreboard for 2x3A:xyi at 30^3, 45.8 ms of the
// 27-k case).  They and the next step's G plane are therefore copied
// asynchronously into slots of shared memory that belong to the reading thread
// alone, so a thread waits for its own copies and the passes' barriers stay the
// only ones (20.3 ms with registers for three sums, 22.4 with their FP64 additions
// every FLUSH sources; 23.0 instead of 20.3 with one CTA more and
// spills).  FP64 planes beyond 32^2 leave no room for the slots: there operands
// are loaded in place and the sums live in shared memory.
// GS > 1: the first GS - 1 outputs of a group wait in registers.
constexpr int MAXSRC = 64;           // sources per chunk (plan_chunks): rows of pencil masks in shared memory
// FP32 sums cover at most FLUSH sources before they go to the FP64 accumulators, so that
// their rounding stays below that of the products they add (a transform of 6 lines and two
// complex products each) however many sources there are.  Against one sum per chunk 8
// cost 2.6 to 3.8% of a mixed pass (27 k-points on 30^3 73.6 -> 76.0 ms, eight atoms on
// 48^3 40.2 -> 41.8), 4 cost 5.5 to 9% (78.9, 43.7).
constexpr int FLUSH = 8;
template <typename V> __device__ __forceinline__ bool flush_due(int si) { return sizeof(V) == 8 && (si + 1) % FLUSH == 0; }

template <class Op, class S, typename V> struct Lay {
    static constexpr int B = S::B;
    static constexpr bool STG = sizeof(V) == 8 || S::N <= 32;     // staged operands, sums in registers
    static constexpr size_t PLANES = sizeof(V) * 2 * (size_t)S::N * S::PAD;
    static constexpr size_t ACC = STG ? 0 : sizeof(V) * (size_t)Op::NACC * B * S::THREADS;
    static constexpr size_t OPS = STG ? sizeof(V) * (size_t)Op::NOPS * B * S::THREADS : 0;
    static constexpr size_t GPL = STG ? sizeof(V) * (size_t)S::N * S::N : 0;
    // registers: in FP32 96 (3 CTAs of 6 warps) with three sums per point, 72 with one
    static constexpr int REGS = sizeof(V) == 8 ? 66 + 2 * Op::NACC * B : (STG ? 108 + 4 * Op::NACC * B : 112);
    // The twiddles come from a table in shared memory where their registers would be spilled
    // (by more than the compiler saves elsewhere): 2x3A on 30^3 4.34 -> 3.33 ms in FP64 (312
    // bytes of spills), 21.9 -> 20.3 ms in FP32 (60 bytes); where they fit the reads cost 1 to
    // 3% (16^3 FP64 1.86 -> 1.90, one sum on 30^3 0.383 -> 0.396).
    // CAP: what launch_bounds leaves a thread (16384 registers per quarter of an SM)
    static constexpr int WARPS = (S::THREADS + 31) / 32 * ctas_for(S::THREADS, REGS);
    static constexpr int CAP = 512 / ((WARPS + 3) / 4) / 8 * 8;
    static constexpr bool TWS = STG && REGS + (int)sizeof(V) / 4 * (S::A + B - 2) > CAP + 16;
    static constexpr size_t TWT = TWS ? sizeof(V) * (size_t)S::N : 0;
    // FP32: the density of re-forwarded planes at the thread's points, read once per CTA (from
    // global memory it cost a wait per source: 48^3 13.4 -> 13.1 ms)
    static constexpr bool RW = STG && sizeof(V) == 8 && Op::REFWD && Op::NRW == 1;
    static constexpr size_t DEN = RW ? sizeof(V) * (size_t)B * S::THREADS : 0;
    static constexpr size_t TOTAL = PLANES + ACC + OPS + GPL + DEN + TWT;
};
template <class Op, class S, typename V> struct Acc {
    static constexpr bool SM = !Lay<Op, S, V>::STG;
    static constexpr int B = S::B;
    V r[SM ? 1 : Op::NACC][SM ? 1 : B];
    V *sm;
    __device__ __forceinline__ V &at(int slot, int m)
    {
        if constexpr (SM) return sm[(slot * B + m) * S::THREADS + threadIdx.x];
        else return r[slot][m];
    }
};

template <typename T, class Op, class S>
__global__ void __launch_bounds__(S::THREADS, ctas_for(S::THREADS, Lay<Op, S, typename C2<T>::t>::REGS)) k_xyi(Op op, int nt)
{
    using V = typename C2<T>::t;
    using L = Lay<Op, S, V>;
    constexpr int N = S::N, A = S::A, B = S::B, PS = S::N * S::PAD, NA = Op::NACC, NO = Op::NOPS;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *b0 = reinterpret_cast<V *>(smem_raw), *b1 = b0 + PS;
    const int t = threadIdx.x / S::LP, l = threadIdx.x % S::LP;
    const bool on = S::LP == N || l < N;
    const int z = blockIdx.x / nt, tj = blockIdx.x % nt;
    const size_t pz = (size_t)z * N * N, p0 = pz + (size_t)t * N + l;
    const int ns = op.nsrc(tj);
    static_assert(!(Op::REFWD && Op::GS > 1), "re-forward needs GS == 1");
    static_assert(Op::NB % Op::GS == 0, "whole output groups");
    Acc<Op, S, V> acc;
    acc.sm = reinterpret_cast<V *>(smem_raw + L::PLANES);
    V *ops = reinterpret_cast<V *>(smem_raw + L::PLANES + L::ACC) + threadIdx.x;            // [NO][B][THREADS]
    V *gpl = reinterpret_cast<V *>(smem_raw + L::PLANES + L::ACC + L::OPS) + t * N + l;     // [A][B][N], t < B
    // pruned chunks: mask of the needed kx per (source, row ky)
    unsigned long long *sbits = reinterpret_cast<unsigned long long *>(smem_raw + L::TOTAL);
    const bool prune = op.m.prune != 0;
    if (prune) {
        for (int i = threadIdx.x; i < ns * N; i += S::THREADS)
            sbits[i] = op.m.pbits[(size_t)op.pent_of(op.item_of(tj, i / N)) * N + i % N];
        __syncthreads();
    }
#pragma unroll
    for (int a = 0; a < NA; a++)
#pragma unroll
        for (int m = 0; m < B; m++) acc.at(a, m) = czero<V>();
    V keep[Op::GS][B];
    V *den = reinterpret_cast<V *>(smem_raw + L::PLANES + L::ACC + L::OPS + L::GPL) + threadIdx.x;
    if constexpr (L::RW) {
        if (on)
#pragma unroll
            for (int m = 0; m < B; m++) den[m * S::THREADS] = __ldg(op.refwd_dens(0) + p0 + (size_t)A * m * N);
    }
    std::conditional_t<L::TWS, TwS<V>, Tw<V, A>> twi;
    std::conditional_t<L::TWS, TwS<V>, Tw<V, B>> twf;
    if constexpr (L::TWS) {
        V *tab = reinterpret_cast<V *>(smem_raw + L::TOTAL - L::TWT);
        for (int i = threadIdx.x; i < N; i += S::THREADS) tab[i] = twsrc<V>(op.g)[i];
        twi = {tab, t < B ? t : 0};
        twf = {tab, t};
        __syncthreads();
    } else {
        twi.load(op.g, t < B ? t : 0);
        if (Op::REFWD) twf.load(op.g, t);
    }
    auto mask = [&](int si, int b) { return prune && ((Op::BLO >> b) & 1) ? sbits[si * N + l] : ~0ull; };
    V nx[L::STG ? 1 : A];
    auto fetch = [&](int si, int b) {
        if (on && t < B) {
            const V *src = op.xyi_grid(op.item_of(tj, si), b) + pz + (size_t)t * N + l;
            const unsigned long long bits = mask(si, b) >> t;
#pragma unroll
            for (int m = 0; m < A; m++) {
                const bool on = (bits >> (B * m)) & 1;
                if constexpr (L::STG) {
                    if (on) fast::cp_async_elem(gpl + m * B * N, src + (size_t)B * m * N);
                } else {
                    nx[m] = on ? src[(size_t)B * m * N] : czero<V>();
                }
            }
        }
        if constexpr (L::STG) cp_commit();
    };
    fetch(0, 0);
    int bg = 0, si = 0, q = 0;
#pragma unroll 1
    while (true) {
        V u[A], v[B];
        if constexpr (L::STG) {
            cp_wait<0>();
            if (on && t < B) {
                const unsigned long long bits = mask(si, bg + q) >> t;
#pragma unroll
                for (int m = 0; m < A; m++) u[m] = (bits >> (B * m)) & 1 ? gpl[m * B * N] : czero<V>();
            }
            if (on && q == Op::GS - 1) {
#pragma unroll
                for (int k = 0; k < NO; k++) {
                    const V *src = op.xyi_operand(k, bg, si);
                    if (src) {
#pragma unroll
                        for (int m = 0; m < B; m++)
                            fast::cp_async_elem(ops + (k * B + m) * S::THREADS, src + p0 + (size_t)A * m * N);
                    }
                }
            }
            cp_commit();
        } else {
#pragma unroll
            for (int m = 0; m < A; m++) u[m] = nx[m];
        }
        // the step after this one: next of the group, next source, next group
        int qn = q + 1, sn = si, bn = bg;
        if (Op::GS == 1 || qn == Op::GS) {
            qn = 0;
            if (++sn == ns) {
                sn = 0;
                bn += Op::GS;
            }
        }
        const bool last = bn == Op::NB;
        if (!last) fetch(sn, bn + qn);
        else if (L::STG) cp_commit();
        plane_inv<V, S>(b0, b1, t, l, u, twi, v);
        {
            V *s = b0;
            b0 = b1;
            b1 = s;
        }
        if (Op::GS > 1 && q < Op::GS - 1) {
#pragma unroll
            for (int m = 0; m < B; m++) keep[q][m] = v[m];
            q = qn;
            continue;
        }
        const int item = op.item_of(tj, si);
        if constexpr (L::STG) cp_wait<1>();      // this step's operands; the next G plane may be on its way
        if (on) {
#pragma unroll
            for (int m = 0; m < B; m++) {
                V vals[Op::GS], o[NO];
#pragma unroll
                for (int g = 0; g < Op::GS - 1; g++) vals[g] = keep[g][m];
                vals[Op::GS - 1] = v[m];
#pragma unroll
                for (int k = 0; k < NO; k++) {
                    if constexpr (L::STG) o[k] = ops[(k * B + m) * S::THREADS];
                    else {
                        const V *src = op.xyi_operand(k, bg, si);
                        o[k] = src ? __ldg(src + p0 + (size_t)A * m * N) : czero<V>();
                    }
                }
                op.xyi_add(si, bg, vals, o, [&](int slot, V x) {
                    V &a = acc.at(slot, m);
                    a = cadd(a, x);
                });
            }
        }
        if (Op::REFWD && op.refwd_want(bg)) {   // uniform over the CTA
            // derived plane (orbital x density): forward XY straight from the registers
            V w[A];
            if (on) {
#pragma unroll
                for (int m = 0; m < B; m++) {
                    if constexpr (L::RW) v[m] = op.refwd_mul(item, v[m], den[m * S::THREADS]);
                    else v[m] = op.refwd_load(tj, item, bg, p0 + (size_t)A * m * N, v[m]);
                }
            }
            plane_fwd<V, S>(b0, b1, t, l, v, twf, w);
            {
                V *s = b0;
                b0 = b1;
                b1 = s;
            }
            if (on && t < B) {
                V *dst = op.refwd_grid(item, bg) + pz + (size_t)t * N + l;
                const unsigned long long bits = (prune ? sbits[si * N + l] : ~0ull) >> t;
#pragma unroll
                for (int m = 0; m < A; m++)
                    if ((bits >> (B * m)) & 1) dst[(size_t)B * m * N] = w[m];
            }
        }
        if (bn != bg || flush_due<V>(si)) {      // the group's last source
            if (on) {
#pragma unroll
                for (int a = 0; a < NA; a++)
#pragma unroll
                    for (int m = 0; m < B; m++) {
                        op.xyi_put(tj, bg, a, p0 + (size_t)A * m * N, acc.at(a, m));
                        acc.at(a, m) = czero<V>();
                    }
            }
            if (last) break;
        }
        bg = bn;
        si = sn;
        q = qn;
    }
}
template <typename V, class S, class Op> __host__ inline size_t smem_xyi(bool prune, int ns)
{
    return Lay<Op, S, V>::TOTAL + (prune ? (size_t)ns * S::N * sizeof(unsigned long long) : 0);
}
// ----------------------------------------------------------------- Z --------
// One item and 32 consecutive pencils per CTA, A threads per z-line, one
// exchange per transform.  The G-space combination is linear: output ZMO (if
// any) is sum_f zmixc(f) X_f, every other output zoutc(o) X_zsrc(o) with
// zsrc(o) < ZK, so only ZK transformed inputs and one sum stay in registers
// (with all inputs of 2x3A kept, 80 registers and 4 CTAs left the pass waiting
// for its loads: issue slots 43% busy, long_scoreboard the main stall).
template <typename T, class Op> __host__ __device__ constexpr bool zk_shared()
{
    return sizeof(T) == 8 && Op::ZINV && Op::NB > (Op::ZMO >= 0 ? 1 : 0);
}
template <typename T, class Op, class S>
__global__ void __launch_bounds__(S::ZTHREADS, ctas_for(S::ZTHREADS, sizeof(T) == 4 ? (Op::NF > 4 ? 96 : 64) : 112)) k_z(Op op)
{
    using V = typename C2<T>::t;
    constexpr int N = S::N, A = S::A, B = S::B, TC = 32, NF = Op::NF, ZK = Op::ZK;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    V *E = reinterpret_cast<V *>(smem_raw);   // [N][TC] exchange buffers, one per input
    const int item = blockIdx.y;
    const int t = threadIdx.x / TC, cl = threadIdx.x % TC;
    // pruning: the CTA takes its 32 pencils from the pair's list (active
    // pencils first); pruned inputs read as zero, pruned outputs are not
    // written off the support
    const bool prune = op.m.prune != 0;
    const int slot = blockIdx.x * TC + cl;
    int c = slot;
    bool allin = false, pon = true;
    if (prune) {
        const int e = op.pent_of(item);
        const int na = op.m.pnact[e];
        if (slot < N * N) c = op.m.pperm[(size_t)e * op.m.np + slot];
        allin = blockIdx.x * TC >= na;
        pon = slot < na;
        constexpr unsigned FI = (1u << NF) - 1, FO = (1u << Op::NB) - 1;
        if (allin && (Op::BLI & FI) == FI && (Op::BLO & FO) == FO) return;   // uniform over the CTA
    }
    const bool act = slot < N * N;
    const auto zc = op.zctx(item, op.m.tr ? c / N : c % N, op.m.tr ? c % N : c / N, c);
    {
        V u[NF][B];
#pragma unroll
        for (int f = 0; f < NF; f++) {
            const bool bl = prune && ((Op::BLI >> f) & 1);
            const V *src = op.zin_grid(item, f) + c;
#pragma unroll
            for (int m = 0; m < B; m++) u[f][m] = (act && (!bl || pon)) ? src[(size_t)(t + A * m) * N * N] : czero<V>();
        }
        Tw<V, B> twf;
        twf.load(op.g, t);
#pragma unroll
        for (int f = 0; f < NF; f++) {
            step1<V, B, -1>(u[f], twf);
            put<V, A, B>(E + f * N * TC + cl, TC, t, u[f]);
        }
    }
    __syncthreads();
    // FP64: the kept inputs go back to the entries of the exchange buffers that only this
    // thread reads (in registers they spilled: 300 to 570 bytes per thread)
    constexpr bool KS = zk_shared<T, Op>();
    V K[KS ? 1 : ZK][KS ? 1 : A], v[A];
    V *const own = E + t * A * TC + cl;
    if (t < B) {
#pragma unroll
        for (int f = 0; f < NF; f++) {
            V X[A];
            step2<V, A, B, -1>(E + f * N * TC + cl, TC, t, X);   // z = t + B m
            if (f < ZK) {
#pragma unroll
                for (int m = 0; m < A; m++) {
                    if constexpr (KS) own[(f * N + m) * TC] = X[m];
                    else K[f < ZK ? f : 0][m] = X[m];
                }
            }
            if constexpr (Op::ZMO >= 0) {
                if (f >= Op::ZM0) {
#pragma unroll
                    for (int m = 0; m < A; m++) {
                        const V w = cscale(X[m], act ? op.zmixc(zc, f, t + B * m) : (T)0);
                        v[m] = f == Op::ZM0 ? w : cadd(v[m], w);
                    }
                }
            }
        }
    }
    Tw<V, A> twi;
    if (Op::ZINV) twi.load(op.g, t < B ? t : 0);
    __syncthreads();                          // the exchange buffers are free
    if constexpr (KS) E += ZK * N * TC;
    int buf = 0;
#pragma unroll 1
    for (int i = 0; i < Op::NB; i++) {
        // the mixed output first: v holds it
        const int o = Op::ZMO > 0 ? (i == 0 ? Op::ZMO : (i <= Op::ZMO ? i - 1 : i)) : i;
        const bool blo = prune && ((Op::BLO >> o) & 1);
        if (blo && allin) continue;       // uniform over the CTA
        if (t < B && (Op::ZMO < 0 || i > 0)) {
            const int k = op.zsrc(o);
#pragma unroll
            for (int m = 0; m < A; m++) {
                const T w = act ? op.zoutc(zc, o, t + B * m) : (T)0;
                if constexpr (KS) v[m] = cscale(own[((ZK > 1 && k ? (ZK - 1) * N : 0) + m) * TC], w);
                else v[m] = cscale(ZK > 1 && k ? K[ZK - 1][m] : K[0][m], w);
            }
        }
        if (Op::ZINV) {
            V *Eo = E + buf * N * TC + cl;
            buf ^= 1;
            if (t < B) {
                step1<V, A, +1>(v, twi);
                put<V, B, A>(Eo, TC, t, v);
            }
            __syncthreads();
            V r[B];
            step2<V, B, A, +1>(Eo, TC, t, r);   // z = t + A m
            if (act && (!blo || pon)) {
                V *dst = op.out_grid(item, o) + c;
#pragma unroll
                for (int m = 0; m < B; m++) dst[(size_t)(t + A * m) * N * N] = r[m];
            }
        } else if (act && t < B && (!blo || pon)) {
            V *dst = op.out_grid(item, o) + c;
#pragma unroll
            for (int m = 0; m < A; m++) dst[(size_t)(t + B * m) * N * N] = v[m];
        }
    }
}
template <typename T, class Op, class S> __host__ inline size_t smem_z()
{
    constexpr int out = zk_shared<T, Op>() ? Op::ZK + 2 : 2, nb = Op::NF > out ? Op::NF : out;
    return sizeof(typename C2<T>::t) * (size_t)nb * S::N * 32;
}

} // namespace sl
} // namespace tcg
