// Bluestein steps in complex128 with a real time step: fixed-point lines.
#include "qsg_blue_inst.cuh"

namespace qsg {

cudaError_t launch_evolve1d_blue_fx(int m, const BlueArgs &a, cudaStream_t st)
{
#define X(T, M) case M: return run_blue<T, M, true>(a, st);
    switch (m) { QSG_BLUE_M(X, double) default: break; }
#undef X
    return cudaErrorNotSupported;
}

cudaError_t launch_kinetic1d_blue_fx(int m, const BlueArgs &a, double dtk, double *sums, cudaStream_t st)
{
#define X(T, M) case M: return run_blue_kin<T, M, true>(a, dtk, sums, st);
    switch (m) { QSG_BLUE_M(X, double) default: break; }
#undef X
    return cudaErrorNotSupported;
}

cudaError_t launch_row_blue_fx(int m, const Blue2DArgs &a, cudaStream_t st)
{
#define X(T, M) case M: return run_row_blue<T, M, true>(a, st);
    switch (m) { QSG_BLUE_M(X, double) default: break; }
#undef X
    return cudaErrorNotSupported;
}

cudaError_t launch_col_blue_fx(int m, const Blue2DArgs &a, bool kinetic, double dtx, double dty, double *partials,
                               cudaStream_t st)
{
#define X(T, M) case M: return run_col_blue<T, M, true>(a, kinetic, dtx, dty, partials, st);
    switch (m) { QSG_BLUE_M(X, double) default: break; }
#undef X
    return cudaErrorNotSupported;
}

}  // namespace qsg
