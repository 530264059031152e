// fast_inst.cu -- explicit instantiation of the fast pass kernels for one cubic
// grid size N = TCG_FAST_N and precision TCG_FAST_T (the build compiles this file
// once per pair).
#include "fast_launch.cuh"
#include "ops_inst.cuh"

#if !defined(TCG_FAST_N) || !defined(TCG_FAST_T)
#error "TCG_FAST_N and TCG_FAST_T must be defined"
#endif

namespace tcg {
#define TCG_INST(T, OP) \
    template int run_chunk_fast<T, TCG_FAST_N, OP>(tcg_ctx *, const OP &, int, int, bool, bool);
TCG_INST_ALL(TCG_FAST_T)
template struct FastIO<TCG_FAST_T, TCG_FAST_N>;
} // namespace tcg
