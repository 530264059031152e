// cube.cu -- instances of the on-chip hf2x kernel (cube.cuh).
#include "cube.cuh"

namespace tcg {
namespace {
template <typename T, int N> int call_n(tcg_ctx *c, const CubeCall<T> &a)
{
    using V = typename C2<T>::t;
    cube::TwN<V, N> tw;
    for (int i = 0; i < N; i++) {
        if constexpr (sizeof(T) == 4) tw.w[i] = c->htw32[i];
        else tw.w[i] = c->htw64[i];
    }
    const double gb = (double)N * N * N * sizeof(V);
    return launch_tagged(c, tagname("hf2x", "cube"), 2.0 * a.nt * a.ns * gb, cube::k_hf<T, N>, dim3(a.nt, a.splits),
                         dim3((N * N + 31) / 32 * 32), cube::smem_hf<T, N>(), a, tw);
}
} // namespace

#define TCG_CUBE_SIZES(X) X(12) X(15) X(16) X(18) X(20)
template <typename T> bool hf_cube_has(int n)
{
#define TCG_C(m) if (n == m && cube::fits<T, m>()) return true;
    TCG_CUBE_SIZES(TCG_C)
#undef TCG_C
    return false;
}
template <typename T> int hf_cube(tcg_ctx *c, const CubeCall<T> &a)
{
    switch (c->fast_n) {
#define TCG_C(m) case m: if constexpr (cube::fits<T, m>()) return call_n<T, m>(c, a); break;
    TCG_CUBE_SIZES(TCG_C)
#undef TCG_C
    default: break;
    }
    return fail(TCG_ERR_UNSUPPORTED, "no on-chip kernel for this grid");
}
template bool hf_cube_has<float>(int);
template bool hf_cube_has<double>(int);
template int hf_cube<float>(tcg_ctx *, const CubeCall<float> &);
template int hf_cube<double>(tcg_ctx *, const CubeCall<double> &);
} // namespace tcg
