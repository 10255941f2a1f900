// 1D evolution in complex128 with a real time step: fixed-point products and lines
// (one CTA, walls, four-step passes).
#include "qsg_evolve1d_inst.cuh"

namespace qsg {

cudaError_t launch_evolve1d_fx(int n, bool few, const Evolve1DBatchArgs &a, cudaStream_t st)
{
#define X(T, L) case L: return few ? run_evolve1d<T, L, true, true>(a, st) : run_evolve1d<T, L, false, true>(a, st);
    switch (n) { QSG_1D_CASES(X, double) default: break; }
#undef X
    return cudaErrorNotSupported;
}

cudaError_t launch_wall1d_fx(int n, const Evolve1DBatchArgs &a, cudaStream_t st)
{
#define X(T, L) case L / 2: return run_wall<T, L, true>(a, st);
    switch (n) { QSG_1D_CASES(X, double) default: break; }
#undef X
    return cudaErrorNotSupported;
}

cudaError_t launch_fs_col_fx(const FsGeom &g, const FsColArgs &a, int ninst, cudaStream_t st)
{
#define X(T, N2) case N2: return run_fs_col<T, N2, true>(g, a, ninst, st);
    switch (g.n2) { QSG_FS_N2(X, double) default: break; }
#undef X
    return cudaErrorNotSupported;
}

cudaError_t launch_fs_row_fx(const FsGeom &g, const FsRowArgs &a, int ninst, cudaStream_t st)
{
#define X(T, N1) case N1: return run_fs_row<T, N1, true>(g, a, ninst, st);
    switch (g.n1) { QSG_FS_N(X, double) default: break; }
#undef X
    return cudaErrorNotSupported;
}

}  // namespace qsg
