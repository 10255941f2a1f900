// qsg_evolve1d_inst.cuh -- launchers of the one-CTA 1D kernels, instantiated by
// qsg_evolve1d.cu, qsg_evolve1d_f32.cu (packed pairs) and qsg_evolve1d_fx.cu (complex128 in
// fixed point), and of the four-step passes.
#pragma once
#include "qsg_dispatch.cuh"

namespace qsg {

// Lines per CTA.  Launches over many lines (batches, the server): 256 threads'
// worth.  Launches of no more than a CTA per SM (`few`): one line or a warp's
// worth, so that short lines do not share an SM with copies of themselves.
constexpr int res_ni_for(int l, int e, bool few)
{
    const int threads = few ? 32 : 256;
    return threads / (l / e) > 1 ? threads / (l / e) : 1;
}
static inline bool res_few(int l, int e, int count) { return count <= res_ni_for(l, e, true) * sm_count(); }

#define QSG_1D_CASES(X, T) \
    X(T, 64) X(T, 128) X(T, 256) X(T, 512) X(T, 1024) X(T, 2048) X(T, 4096)

// complex64 walls (lines of L = 2n): in packed pairs where the last stage is of
// radix 4 or 8, scalar where all stages are of radix 16 (and one of 2).  Scalar to
// packed, us per O4 step: n = 64 4.10 -> 3.83, 512 5.99 -> 5.72, 1024 7.47 -> 7.04;
// 128 3.99 -> 4.26, 256 5.84 -> 6.00, 2048 11.29 -> 11.77, 4096 31.3 -> 31.8.
#define QSG_WALL_PACKED(X, T) X(T, 128) X(T, 1024) X(T, 2048)
#define QSG_WALL_SCALAR(X, T) X(T, 256) X(T, 512) X(T, 4096) X(T, 8192)

template <class T, int L, bool FEW, bool FX = false>
static cudaError_t run_evolve1d(const Evolve1DBatchArgs &a, cudaStream_t st)
{
    constexpr int E = sizeof(T) == 4 ? 16 : 8;
    constexpr int PADS = sizeof(T) == 4 ? 4 : 3;
    constexpr int NI = res_ni_for(L, E, FEW);
    const size_t smem = sizeof(cplx_t<T>) * padded<L, PADS>(L) * NI;
    auto k = k_evolve1d_resident<T, L, E, NI, FX>;
    cudaError_t e = prepare_smem(k, smem);
    if (e != cudaSuccess) return e;
    launch_pdl(k, dim3((a.count + NI - 1) / NI), dim3(NI * (L / E)), smem, st, a);
    return cudaGetLastError();
}

template <class T, int L2, bool FX = false>
static cudaError_t run_wall(const Evolve1DBatchArgs &a, cudaStream_t st)
{
    constexpr int E = sizeof(T) == 4 ? 16 : 8;
    constexpr int PADS = sizeof(T) == 4 ? 4 : 3;
    const size_t smem = sizeof(cplx_t<T>) * padded<L2, PADS>(L2);
    auto k = k_evolve1d_wall<T, L2, E, FX>;
    cudaError_t e = prepare_smem(k, smem);
    if (e != cudaSuccess) return e;
    launch_pdl(k, dim3(a.count), dim3(L2 / E), smem, st, a);
    return cudaGetLastError();
}

// four-step passes: columns per column-pass CTA, rows per row-pass CTA
constexpr int fs_col_w(int prec, int n2) { return prec == 1 ? 4096 / n2 : 2048 / n2; }   // W*n2/E = 256
constexpr int fs_row_b(int prec, int n1)   // B*n1/E = 256 (512 for complex128 rows of 4096)
{
    return prec == 1 ? 4096 / n1 : (n1 >= 2048 ? 1 : 2048 / n1);
}

template <class T, int N2, bool FX = false>
static cudaError_t run_fs_col(const FsGeom &g, const FsColArgs &a, int ninst, cudaStream_t st)
{
    constexpr int P = sizeof(T) == 4 ? 1 : 0;
    constexpr int E = P ? 16 : 8;
    constexpr int W = fs_col_w(P, N2);
    auto k = k_fs_col<T, N2, E, W, FX>;
    cudaError_t e = prepare_smem(k, g.col_smem);
    if (e != cudaSuccess) return e;
    launch_pdl(k, dim3(g.col_blocks, ninst), dim3(W * (N2 / E)), g.col_smem, st, a);
    return cudaGetLastError();
}

template <class T, int N1, bool FX = false>
static cudaError_t run_fs_row(const FsGeom &g, const FsRowArgs &a, int ninst, cudaStream_t st)
{
    constexpr int P = sizeof(T) == 4 ? 1 : 0;
    constexpr int E = P ? 16 : 8;
    constexpr int B = fs_row_b(P, N1);
    auto k = k_fs_row<T, N1, E, B, FX>;
    cudaError_t e = prepare_smem(k, g.row_smem);
    if (e != cudaSuccess) return e;
    launch_pdl(k, dim3(g.row_blocks, ninst), dim3(B * (N1 / E)), g.row_smem, st, a);
    return cudaGetLastError();
}

#define QSG_FS_N(X, T) X(T, 64) X(T, 128) X(T, 256) X(T, 512) X(T, 1024) X(T, 2048) X(T, 4096)
#define QSG_FS_N2(X, T) X(T, 64) X(T, 128) X(T, 256) X(T, 512) X(T, 1024) X(T, 2048)

cudaError_t launch_evolve1d_few_f32(int n, const Evolve1DBatchArgs &a, cudaStream_t st);
cudaError_t launch_wall1d_f32(int n, const Evolve1DBatchArgs &a, cudaStream_t st);
cudaError_t launch_evolve1d_fx(int n, bool few, const Evolve1DBatchArgs &a, cudaStream_t st);
cudaError_t launch_wall1d_fx(int n, const Evolve1DBatchArgs &a, cudaStream_t st);
cudaError_t launch_fs_col_fx(const FsGeom &g, const FsColArgs &a, int ninst, cudaStream_t st);
cudaError_t launch_fs_row_fx(const FsGeom &g, const FsRowArgs &a, int ninst, cudaStream_t st);

}  // namespace qsg
