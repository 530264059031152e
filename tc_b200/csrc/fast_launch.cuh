// fast_launch.cuh -- launcher of the compile-time-size pass kernels (cubic
// grids).  Algorithmic bytes per launch as in run_chunk: N s per grid and pass.
#pragma once
#include "terms.cuh"
#include "fast.cuh"
#include "split.cuh"
#include "fft_split.cuh"

namespace tcg {

template <typename T, int N, class Op>
int run_chunk_fast(tcg_ctx *c, const Op &op, int items, int nt, bool do_xyf, bool do_xyi)
{
    using V = typename C2<T>::t;
    using CF = fast::Cfg<N, sizeof(V)>;
    const double gb = (double)N * N * N * sizeof(V);
    // bytes a pass must move: N s per grid, the band-limited grids of a pruned
    // chunk only on the pencils their support meets (fraction op.m.pfrac)
    const double fr = op.m.prune ? op.m.pfrac : 1.0;
    const int bli = __builtin_popcount(Op::BLI), blo = __builtin_popcount(Op::BLO);
    const double nf_eff = (Op::NF - bli) + fr * bli, nb_eff = (Op::NB - blo) + fr * blo;
    const int np_f = items * N, np_i = nt * N;
    const bool slx = split_xy(c), slz = split_z(c);
    using SH = sl::Shape<N, sl::ShapeOf<N>::A, sl::ShapeOf<N>::B>;
    const int nref = Op::REFWD ? Op::NB - 1 : 0;
    if (slx && do_xyf) {
        const double by = (double)items * nf_eff * gb;
        if constexpr (Op::NSO == 0) {
            TRY(launch_tagged(c, tagname(Op::NAME, "xyf"), by, sl::k_xyf_items<T, Op, SH>, dim3(np_f), dim3(SH::THREADS),
                              sl::smem_xyf<V, SH, Op>(), op, items));
        } else {
            // sources per CTA: at least 8 CTAs per SM and round of 4 where the chunk has them
            const int parts = std::max(1, std::min(op.ns, (148 * 8 * 4 + np_i - 1) / np_i)), per = (op.ns + parts - 1) / parts;
            TRY(launch_tagged(c, tagname(Op::NAME, "xyf"), by, sl::k_xyf<T, Op, SH>, dim3(np_i, (op.ns + per - 1) / per),
                              dim3(SH::THREADS), sl::smem_xyf<V, SH, Op>(), op, nt, per));
        }
    }
    auto z_split = [&]() -> int {
        // pencils nobody needs get no CTA
        const unsigned fi = (1u << Op::NF) - 1, fo = (1u << Op::NB) - 1;
        const bool bl = op.m.prune && (Op::BLI & fi) == fi && (Op::BLO & fo) == fo;
        const int np = bl ? op.m.pmax : N * N;
        return launch_tagged(c, tagname(Op::NAME, "z"), (double)items * (nf_eff + (Op::ZINV ? nb_eff : 0)) * gb,
                             sl::k_z<T, Op, SH>, dim3((np + 31) / 32, items), dim3(SH::ZTHREADS),
                             sl::smem_z<T, Op, SH>(), op);
    };
    if (slx && slz) {
        TRY(z_split());
        if (!do_xyi) return TCG_OK;
        return launch_tagged(c, tagname(Op::NAME, "xyi"), (double)items * (nb_eff + fr * nref) * gb, sl::k_xyi<T, Op, SH>,
                             dim3(np_i), dim3(SH::THREADS),
                             sl::smem_xyi<V, SH, Op>(op.m.prune, op.ns), op, nt);
    }
    if constexpr (line_grid(N)) {
    using CP = fast::CfgP<N, sizeof(V)>;
    const bool fpair = c->xy_kernels ? c->xy_kernels == 2 : Op::XYF_PAIR;
    const bool ipair = c->xy_kernels ? c->xy_kernels == 2 : Op::XYI_PAIR;
    if (do_xyf && !slx) {
        if (!fpair)
            TRY(launch_tagged(c, tagname(Op::NAME, "xyf"), (double)items * Op::NF * gb, fast::k_xyf_fast<T, N, Op>,
                              dim3((np_f + CF::P - 1) / CF::P), dim3(CF::THREADS), fast::smem_xy_fast<V, N>(1), op, np_f));
        else
            TRY(launch_tagged(c, tagname(Op::NAME, "xyf"), (double)items * Op::NF * gb, fast::k_xyf_pair<T, N, Op>,
                              dim3((np_f + CP::P - 1) / CP::P), dim3(CP::THREADS), fast::smem_xy_pair<V, N>(1), op, np_f));
    }
    constexpr int TC = fast::zcols<V>();
    const bool zsplit = c->z_kernels ? c->z_kernels == 2 : Op::ZSPLIT;
    if (slz) TRY(z_split());
    else if (zsplit)
        TRY(launch_tagged(c, tagname(Op::NAME, "z"), (double)items * (Op::NF + (Op::ZINV ? Op::NB : 0)) * gb,
                          fast::k_z_fast<T, N, Op>, dim3((N * N + TC - 1) / TC, items), dim3(128),
                          fast::smem_z_fast<V, N>(Op::NF), op));
    else
        TRY(launch_tagged(c, tagname(Op::NAME, "z"), (double)items * (Op::NF + (Op::ZINV ? Op::NB : 0)) * gb,
                          fast::k_z_line<T, N, Op>, dim3((N * N + TC - 1) / TC, items), dim3(32 * fast::ZL),
                          fast::smem_z_fast<V, N>(Op::NF), op));
    if (slx && do_xyi)
        return launch_tagged(c, tagname(Op::NAME, "xyi"), (double)items * (nb_eff + nref) * gb, sl::k_xyi<T, Op, SH>,
                             dim3(np_i), dim3(SH::THREADS), sl::smem_xyi<V, SH, Op>(false, op.ns), op, nt);
    if (do_xyi) {
        if constexpr (Op::GS == 1 && !(Op::REGACC && Op::REFWD)) {
            if (!ipair && !c->no_prefetch)
                return launch_tagged(c, tagname(Op::NAME, "xyi"), (double)items * (Op::NB + nref) * gb,
                                     fast::k_xyi_pf<T, N, Op>, dim3((np_i + CF::P - 1) / CF::P), dim3(CF::THREADS),
                                     fast::smem_xy_fast<V, N>(2), op, np_i);
        }
        if (!ipair)
            TRY(launch_tagged(c, tagname(Op::NAME, "xyi"), (double)items * (Op::NB + nref) * gb, fast::k_xyi_fast<T, N, Op>,
                              dim3((np_i + CF::P - 1) / CF::P), dim3(CF::THREADS), fast::smem_xy_fast<V, N>(2), op, np_i));
        else
            TRY(launch_tagged(c, tagname(Op::NAME, "xyi"), (double)items * (Op::NB + nref) * gb, fast::k_xyi_pair<T, N, Op>,
                              dim3((np_i + CP::P - 1) / CP::P), dim3(CP::THREADS), fast::smem_xy_pair<V, N>(2), op, np_i));
    }
    }
    return TCG_OK;
}

// ---- whole transforms (fft_split.cuh)
template <int N> using IOShape = sl::Shape<N, sl::ShapeOf<N>::A, sl::ShapeOf<N>::B>;
template <typename T, int N> int FastIO<T, N>::xy(tcg_ctx *c, const GridDesc &g, const GridRefs &gr, unsigned n, int dir)
{
    using V = typename C2<T>::t;
    using S = IOShape<N>;
    return launch(c, dir < 0 ? sl::k_xy_io<T, S, -1> : sl::k_xy_io<T, S, +1>, dim3(N, n), dim3(S::THREADS), sl::smem_xy_io<V, S>(), g,
                  gr);
}
template <typename T, int N>
int FastIO<T, N>::z(tcg_ctx *c, const GridDesc &g, const GridRefs &gr, unsigned n, int dir, double scale)
{
    using V = typename C2<T>::t;
    using S = IOShape<N>;
    return launch(c, dir < 0 ? sl::k_z_io<T, S, -1> : sl::k_z_io<T, S, +1>, dim3((N * N + 31) / 32, n), dim3(S::ZTHREADS),
                  sl::smem_z_io<V, S>(), g, gr, (T)scale);
}
template <typename T, int N> int FastIO<T, N>::sphere(tcg_ctx *c, const GridDesc &g, const SphereItem *items, unsigned n)
{
    using V = typename C2<T>::t;
    using S = IOShape<N>;
    return launch(c, sl::k_sphere_io<T, S>, dim3((N * N + 31) / 32, n), dim3(S::ZTHREADS), sl::smem_z_io<V, S>(), g, items,
                  c->recip.as<const double>());
}
template <typename T, int N> int FastIO<T, N>::gather(tcg_ctx *c, const GridDesc &g, const GatherItem *items, unsigned n)
{
    if constexpr (sizeof(T) == 8) {
        using S = IOShape<N>;
        return launch(c, sl::k_gather_io<S>, dim3((N * N + 31) / 32, n), dim3(S::ZTHREADS), sl::smem_z_io<double2, S>(), g, items);
    } else return fail(TCG_ERR_UNSUPPORTED, "accumulators are double precision");
}

} // namespace tcg
