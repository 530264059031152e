// any_inst.cu -- launcher and instances of the run-time-shape passes
// (anygrid.cuh) for precision TCG_FAST_T (the build compiles this file once per
// precision).  Algorithmic bytes per launch as in run_chunk.
#include "anygrid.cuh"
#include "ops_inst.cuh"

namespace tcg {
template <typename T, class Op>
int run_chunk_any(tcg_ctx *c, const Op &op, int items, int nt, bool do_xyf, bool do_xyi)
{
    using V = typename C2<T>::t;
    const sl::AnyShape &s = c->any;
    const double gb = (double)c->gd.N * sizeof(V), fr = op.m.prune ? op.m.pfrac : 1.0;
    const int bli = __builtin_popcount(Op::BLI), blo = __builtin_popcount(Op::BLO), nref = Op::REFWD ? Op::NB - 1 : 0;
    const double nf = (Op::NF - bli) + fr * bli, nb = (Op::NB - blo) + fr * blo;
    const int thr = std::max(s.a[1] * s.n[0], s.a[0] * s.n[1]), np = s.n[0] * s.n[1];
    const size_t xy = sizeof(V) * (s.n[0] + s.n[1] + 2 * (size_t)s.ps);
    auto xyf = thr <= 256 ? anyg::k_xyf<T, Op, 256> : anyg::k_xyf<T, Op, sl::MAXTHR>;
    auto xyi = thr <= 256 ? anyg::k_xyi<T, Op, 256> : anyg::k_xyi<T, Op, sl::MAXTHR>;
    if (do_xyf)
        TRY(launch_tagged(c, tagname(Op::NAME, "xyf"), items * nf * gb, xyf, dim3(items * s.n[2]), dim3(thr), xy, op, s, items));
    const unsigned fi = (1u << Op::NF) - 1, fo = (1u << Op::NB) - 1;
    const bool bl = op.m.prune && (Op::BLI & fi) == fi && (Op::BLO & fo) == fo;
    TRY(launch_tagged(c, tagname(Op::NAME, "z"), items * (nf + (Op::ZINV ? nb : 0)) * gb, anyg::k_z<T, Op>,
                      dim3(((bl ? op.m.pmax : np) + 31) / 32, items), dim3(32 * s.a[2]),
                      sizeof(V) * (size_t)s.n[2] * (1 + 32 * std::max(2, Op::NF)), op, s));
    if (do_xyi)
        TRY(launch_tagged(c, tagname(Op::NAME, "xyi"), items * (nb + fr * nref) * gb, xyi, dim3(nt * s.n[2]), dim3(thr),
                          xy + sizeof(V) * (size_t)Op::NACC * s.b[1] * thr, op, s, nt));
    return TCG_OK;
}
#define TCG_INST(T, OP) template int run_chunk_any<T, OP>(tcg_ctx *, const OP &, int, int, bool, bool);
TCG_INST_ALL(TCG_FAST_T)
} // namespace tcg
