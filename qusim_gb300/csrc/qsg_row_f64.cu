// 2D row passes (double): instantiations + launchers, fixed-point products here and
// double ones (complex time steps) in qsg_row_f64_double.cu, which includes this.
#include "qsg_dispatch.cuh"

namespace qsg {

template <int NY, int E, int G, int NT, bool FX>
static cudaError_t run_row_f64(const Geom2D &g, const RowPassArgs &a, cudaStream_t st)
{
    constexpr int B = row_b_for(NY, E, G, NT);
    constexpr int RS = row_work_for(NY, E, G, NT) / NT;
    static_assert(RS * NT == row_work_for(NY, E, G, NT), "NT must divide the CTA's line work");
    auto k = k_row_pass<double, NY, E, G, B, RS, false, FX>;
    cudaError_t e = prepare_smem(k, g.row_smem);
    if (e != cudaSuccess) return e;
    static int occ = 0;
    launch_pdl(k, dim3(persistent_grid(k, NT, g.row_smem, a.units, occ)), dim3(NT), g.row_smem, st, a);
    return cudaGetLastError();
}

template <bool FX> cudaError_t launch_row_pass_f64_t(const Geom2D &g, const RowPassArgs &a, cudaStream_t st)
{
#define X(T, NY, E, G, NT) \
    if (g.ny == NY && g.row_e == E && g.g == G && g.row_threads == NT) return run_row_f64<NY, E, G, NT, FX>(g, a, st);
    QSG_ROW_VARIANTS_F64(X)
#undef X
    return cudaErrorNotSupported;
}

#ifndef QSG_DOUBLE_UNIT
template cudaError_t launch_row_pass_f64_t<true>(const Geom2D &, const RowPassArgs &, cudaStream_t);

bool row_variant_exists_f64(int ny, int e, int g, int nt)
{
#define X(T, NY, E, G, NT) \
    if (ny == NY && e == E && g == G && nt == NT) return true;
    QSG_ROW_VARIANTS_F64(X)
#undef X
    return false;
}

#else
template cudaError_t launch_row_pass_f64_t<false>(const Geom2D &, const RowPassArgs &, cudaStream_t);
#endif

}  // namespace qsg
