// qsg_blue_inst.cuh -- launchers of the Bluestein kernels, instantiated by
// qsg_blue.cu and qsg_blue_fx.cu (complex128 in fixed point).
#pragma once
#include "qsg_blue.cuh"
#include "qsg_dispatch.cuh"

namespace qsg {

#define QSG_BLUE_M(X, T) X(T, 256) X(T, 512) X(T, 1024) X(T, 2048) X(T, 4096) X(T, 8192)

template <class T, int M, bool FX = false>
static cudaError_t run_blue(const BlueArgs &a, cudaStream_t st)
{
    constexpr int E = FX ? blue_fx_e(M) : (sizeof(T) == 4 ? 16 : 8);
    constexpr int PADS = sizeof(T) == 4 ? 4 : 3;
    const size_t smem = sizeof(cplx_t<T>) * padded<M, PADS>(M);
    auto k = k_evolve1d_blue<T, M, E, FX>;
    cudaError_t e = prepare_smem(k, smem);
    if (e != cudaSuccess) return e;
    launch_pdl(k, dim3(1), dim3(M / E), smem, st, a);
    return cudaGetLastError();
}

template <class T, int M, bool FX = false>
static cudaError_t run_blue_kin(const BlueArgs &a, double dtk, double *sums, cudaStream_t st)
{
    constexpr int E = sizeof(T) == 4 ? 16 : 8;
    constexpr int PADS = sizeof(T) == 4 ? 4 : 3;
    const size_t smem = sizeof(cplx_t<T>) * padded<M, PADS>(M);
    auto k = k_kinetic1d_blue<T, M, E, FX>;
    cudaError_t e = prepare_smem(k, smem);
    if (e != cudaSuccess) return e;
    k<<<1, M / E, smem, st>>>(a, dtk, sums);
    return cudaGetLastError();
}

template <class T, int M, bool FX = false>
static cudaError_t run_row_blue(const Blue2DArgs &a, cudaStream_t st)
{
    constexpr int E = sizeof(T) == 4 ? 16 : 8;
    constexpr int PADS = sizeof(T) == 4 ? 4 : 3;
    constexpr int RPC = (256 / (M / E)) > 1 ? 256 / (M / E) : 1;
    const size_t smem = sizeof(cplx_t<T>) * padded<M, PADS>(M) * RPC;
    auto k = k_row_blue<T, M, E, RPC, FX>;
    cudaError_t e = prepare_smem(k, smem);
    if (e != cudaSuccess) return e;
    launch_pdl(k, dim3((a.nx + RPC - 1) / RPC), dim3(RPC * (M / E)), smem, st, a);
    return cudaGetLastError();
}

template <class T, int M> constexpr int col_w_of()
{
    constexpr int w = 65536 / (M * (int)sizeof(cplx_t<T>));
    return w < 1 ? 1 : (w > 16 ? 16 : w);
}

template <class T, int M, bool FX = false>
static cudaError_t run_col_blue(const Blue2DArgs &a, bool kinetic, double dtx, double dty, double *partials,
                                cudaStream_t st)
{
    constexpr int E = sizeof(T) == 4 ? 16 : 8;
    constexpr int W = col_w_of<T, M>();
    const size_t smem = sizeof(cplx_t<T>) * col_tile_elems(sizeof(cplx_t<T>), M, W);
    const unsigned grid = (unsigned)((a.ny + W - 1) / W);
    if (kinetic) {
        auto k = k_col_blue_kinetic<T, M, E, W, FX>;
        cudaError_t e = prepare_smem(k, smem);
        if (e != cudaSuccess) return e;
        k<<<grid, W * (M / E), smem, st>>>(a, dtx, dty, partials);
    } else {
        auto k = k_col_blue<T, M, E, W, FX>;
        cudaError_t e = prepare_smem(k, smem);
        if (e != cudaSuccess) return e;
        launch_pdl(k, dim3(grid), dim3(W * (M / E)), smem, st, a);
    }
    return cudaGetLastError();
}

cudaError_t launch_evolve1d_blue_fx(int m, const BlueArgs &a, cudaStream_t st);
cudaError_t launch_kinetic1d_blue_fx(int m, const BlueArgs &a, double dtk, double *sums, cudaStream_t st);
cudaError_t launch_row_blue_fx(int m, const Blue2DArgs &a, cudaStream_t st);
cudaError_t launch_col_blue_fx(int m, const Blue2DArgs &a, bool kinetic, double dtx, double dty, double *partials,
                               cudaStream_t st);

}  // namespace qsg
