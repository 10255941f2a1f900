// qsg_evolve1d_inst.cuh -- launchers of the one-CTA 1D kernels, instantiated by
// qsg_evolve1d.cu and qsg_evolve1d_f32.cu (packed pairs).
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

template <class T, int L, bool FEW, bool FX = false>
static cudaError_t run_evolve1d(const Evolve1DBatchArgs &a, cudaStream_t st)
{
    if constexpr (sizeof(T) == 8 && !FX) {
        if (a.fx) return run_evolve1d<T, L, FEW, true>(a, st);
    }
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
    if constexpr (sizeof(T) == 8 && !FX) {
        if (a.fx) return run_wall<T, L2, true>(a, st);
    }
    constexpr int E = sizeof(T) == 4 ? 16 : 8;
    constexpr int PADS = sizeof(T) == 4 ? 4 : 3;
    const size_t smem = sizeof(cplx_t<T>) * padded<L2, PADS>(L2);
    auto k = k_evolve1d_wall<T, L2, E, FX>;
    cudaError_t e = prepare_smem(k, smem);
    if (e != cudaSuccess) return e;
    launch_pdl(k, dim3(a.count), dim3(L2 / E), smem, st, a);
    return cudaGetLastError();
}

cudaError_t launch_evolve1d_few_f32(int n, const Evolve1DBatchArgs &a, cudaStream_t st);
cudaError_t launch_wall1d_f32(int n, const Evolve1DBatchArgs &a, cudaStream_t st);

}  // namespace qsg
