// One-CTA 1D evolution in complex64 where a launch has at most a CTA per SM (a
// line of its own, small batches), and the walls of QSG_WALL_PACKED.  Packed FP32
// pairs: a CTA alone on its SM has the registers (up to 244 per thread), and its
// step is bound by the instructions it issues (with the CTAs of one line, per O2
// step: n = 64 1.84 -> 1.27 us, 1024 3.35 -> 1.53, 4096 4.36 -> 3.28).  Launches
// over more lines, the tile queue and the four-step passes stay scalar in
// qsg_evolve1d.cu: under their register caps the pairs spill (queue of 256 ..
// 2048-site lines 614 -> 1122 us per 100 steps).  Both round alike.
#define QSG_PACKED_F32
#include "qsg_evolve1d_inst.cuh"

namespace qsg {

cudaError_t launch_evolve1d_few_f32(int n, const Evolve1DBatchArgs &a, cudaStream_t st)
{
#define X(T, L) case L: return run_evolve1d<T, L, true>(a, st);
    switch (n) { QSG_1D_CASES(X, float) X(float, 8192) default: break; }
#undef X
    return cudaErrorNotSupported;
}

cudaError_t launch_wall1d_f32(int n, const Evolve1DBatchArgs &a, cudaStream_t st)
{
#define X(T, L) case L / 2: return run_wall<T, L>(a, st);
    switch (n) { QSG_WALL_PACKED(X, float) default: break; }
#undef X
    return cudaErrorNotSupported;
}

}  // namespace qsg
