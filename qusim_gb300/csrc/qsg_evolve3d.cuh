// qsg_evolve3d.cuh -- 3D split-operator passes.
//
// The reference has a 3D transform (KissFourierTransform3D,
// src/FourierTransform.cpp:379-440; z contiguous, index (ix*ny + iy)*nz + iz)
// and a 3D kinetic multiply (MulExpK3D, src/DeviceTemplate.h:851-879), but no 3D
// evolver; this is SplittingMethod2D's step (src/SplittingMethod2D.cpp:38-121)
// with a third axis.  The kinetic factor exp(a (kx^2 DTx + ky^2 DTy + kz^2 DTz))
// is a product of one factor per axis, so the kinetic operator is the product
// of three commuting one-axis operators F_a^-1 K_a F_a: each is a pass over the
// lines along its axis (transform, factor, inverse transform, all on chip), and
// V multiplies fuse into the passes.  A step never leaves natural real-space
// layout.  Because the axes commute, a kinetic substep may take them in any
// order.  An order-4 step takes z y x, x z y, y x z: each substep starts on the
// axis that the one before it ended on, the next step too, and the last axis of
// one, the V between and the same axis of the next are one pass of four
// transforms:
//
//   O4: z[V1 V1', K1] y[K1] x[K1, V2, K2] z[K2] y[K2, V2, K1] x[K1] (z[K1, V1])
//       6 passes a step, and one more that closes a call
//   O2: z[V V', K] y[K] x[K, (V)]
//       3 passes: one substep cannot start and end on the same axis
//
// (V' = the previous step's closing factor; in O4 its pass is also the previous
// step's last, z[K1, V1', V1, K1]; (.) only at a call's end.)  Every step is the
// same sequence of operations on the state wherever a call begins or ends, so
// calls that split a run leave the state of one call bit for bit.  (Orders that
// alternate between z y x and x y z would join O2 steps too, 2 passes a step, but
// then a step's rounding depends on how many came before it: 226 against 243 us
// a step at 256^3 complex64, 1.28 against 1.37 ms complex128, 8.4 against 11.1 at
// 32^3.)  O4 against nine passes of one axis each, per step of 256^3: complex64
// 778 -> 618 us, complex128 with the products in fixed point as well 16.6 -> 3.69
// ms.
// z lines are contiguous (k3_row); y and x lines are strided by nz and ny*nz
// (k3_col, W adjacent z positions per CTA so every access is a W-wide contiguous
// segment).
#pragma once
#include "qsg_kernels.cuh"

namespace qsg {

struct Pass3Args {
    void *psi;
    const void *v[2];      // V factor before the axis operator and after it (or null each; with a
                           // second axis factor the one between the two, not null); natural layout,
                           // n entries
    int v_twice;           // the two ExpV calls at a step boundary: v[1] applied twice where there is a
                           // second axis factor, v[0] otherwise (not with FX)
    const void *k, *k2;    // the axis factor, and a second one (or null): complex64 factor - 1,
                           // complex128 factor / L (FX: fixed-point factors)
    int fx;
    size_t n;              // sites (FX: the V tables' flag entry)
    const void *tw;        // stage twiddles (L, E)
    float inv_l;           // 1/L (complex64)
    long long s_line;      // stride between a line's elements (strided kernel)
    long long s_outer;     // stride between line groups (strided kernel)
    double *partials;      // kinetic mode: 2 per CTA, sum |X|^2 fold(k)^2 and sum |X|^2
    int kinetic;           // 1: forward transform and the kinetic sums only (no store)
};

template <class C, int E, class I> __device__ __forceinline__ void v3_apply(C (&x)[E], const void *v, I idx, bool twice)
{
    const C *vt = opaque(static_cast<const C *>(v));
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const C m = ld_stream(vt + idx(e));
        x[e] = PhaseOps<C>::apply(x[e], m);
        if (twice) x[e] = PhaseOps<C>::apply(x[e], m);
    }
}

// x * K[k] (with 1/L): complex64 cmul1p on the factor - 1 table
template <class C> __device__ __forceinline__ C k3_apply(C x, const C *kt, int k, float inv_l)
{
    if constexpr (sizeof(C) == 8) return cmul1p(cscale(x, inv_l), ld_c(kt + k));
    else return cmul(x, ld_c(kt + k));
}

// [V] F^-1 K F [V] [F^-1 K2 F] on a line in registers, the inverse as
// conj(F(conj(.))); idx(e): the site of slot e.  One transform body in a loop.
// FX (complex128, real time steps): the line is in fixed point throughout.
template <class C, int L, int E, bool FX, class Lay, class Bar, class I>
__device__ __forceinline__ void axis_ops(C (&x)[E], C *sm, const Lay &lay, const Bar &bar, int t, const stw_t<C> *tw,
                                         const Pass3Args &a, I idx)
{
    constexpr int TL = L / E;
    const int nq = a.k2 ? 4 : 2;
    if constexpr (FX) {
        FixLine<L, E> f;
        f.load(x, sm, lay, bar, t);
        auto mul_v = [&](const void *v, bool twice) {
            const fixw *vt = opaque(static_cast<const fixw *>(v));
            if (fix_flagged(vt + a.n)) f.finite = false;
            f.mul_v([&](int e) { return ld_stream(vt + idx(e)); });
            if (twice) {  // between two steps: rounded as a call's end would
                f.round(x, sm, lay, bar, t);
                f.mul_v([&](int e) { return ld_stream(vt + idx(e)); });
            }
        };
        if (a.v[0]) mul_v(a.v[0], false);
#pragma unroll 1
        for (int q = 0; q < nq; ++q) {
            f.fft(sm, lay, bar, t, opaque(tw));
            f.scale(sm, lay, bar, t);
            if ((q & 1) == 0) {
                const fixw *kt = static_cast<const fixw *>(q ? a.k2 : a.k);
                f.ex -= Plan<L, E>::LOGL;  // 1/L
                f.mul([&](int e) { return __ldg(kt + t + e * TL); });
                f.conj();
            } else {
                f.conj();
                if (q == 1 && a.v[1]) mul_v(a.v[1], a.v_twice);
            }
        }
        f.store(x);
    } else {
        if (a.v[0]) v3_apply(x, a.v[0], idx, a.v_twice && !a.k2);
#pragma unroll 1
        for (int q = 0; q < nq; ++q) {
            line_fft<C, L, E, false>(x, sm, lay, bar, t, tw);
            if ((q & 1) == 0) {
                const C *kt = static_cast<const C *>(q ? a.k2 : a.k);
#pragma unroll
                for (int e = 0; e < E; ++e) x[e] = cconj(k3_apply(x[e], kt, t + e * TL, a.inv_l));
            } else {
#pragma unroll
                for (int e = 0; e < E; ++e) x[e] = cconj(x[e]);
                if (q == 1 && a.v[1]) v3_apply(x, a.v[1], idx, a.v_twice && a.k2);
            }
        }
    }
}

// B contiguous lines (z) of L per CTA
// strided passes: three 256-thread CTAs per SM (registers capped at 85), as
// they are bound by the latency of their scattered loads, not by issue
constexpr int min_blocks3(int threads) { return threads <= 256 ? 3 : 1; }
// contiguous lines: the same, except lines within a warp, whose loads the
// compiler schedules across __syncwarp: at 85 registers they spill 270 bytes (z
// of 256^3 150 us a pass of four transforms, 131 with two CTAs per SM)
constexpr int min_blocks3_row(int threads, int tl) { return threads > 256 ? 1 : (tl <= 32 ? 2 : 3); }

template <class T, int L, int E, int B, bool FX = false>
__global__ void __launch_bounds__(B *(L / E), min_blocks3_row(B *(L / E), L / E)) k3_row(Pass3Args a)
{
    pdl_wait();
    using C = cplx_t<T>;
    constexpr int TL = Plan<L, E>::TL;
    constexpr int NT = B * TL;
    constexpr int PADS = sizeof(C) == 8 ? 4 : 3;
    constexpr int LINE = padded<L, PADS>(L);
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[32];
    C *sm = reinterpret_cast<C *>(smraw);
    const int tid = threadIdx.x;
    const int line = tid / TL, t = tid - line * TL;
    const size_t base = ((size_t)blockIdx.x * B + line) * L + t;
    const RowLayout<PADS> lay{line * LINE};
    const auto lbar = LineBarrierOf<TL, B>::make(line);
    C *psi = static_cast<C *>(a.psi);
    const stw_t<C> *tw = static_cast<const stw_t<C> *>(a.tw);

    C x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = ld_stream(psi + base + e * TL);
    if (a.kinetic) {
        line_fft<C, L, E, false>(x, sm, lay, lbar, t, tw);
        double s1 = 0, s0 = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int k = t + e * TL;
            const double f = (double)(k > L / 2 ? L - k : k);
            const double m = abs2d(x[e]);
            s1 += m * f * f;
            s0 += m;
        }
        s1 = block_sum<NT>(s1, red);
        s0 = block_sum<NT>(s0, red);
        if (tid == 0) {
            a.partials[2 * blockIdx.x] = s1;
            a.partials[2 * blockIdx.x + 1] = s0;
        }
        return;
    }
    axis_ops<C, L, E, FX>(x, sm, lay, lbar, t, tw, a, [=](int e) { return base + e * TL; });
    C *o = const_cast<C *>(opaque(psi));
#pragma unroll
    for (int e = 0; e < E; ++e) st_stream(o + base + e * TL, x[e]);
}

// strided lines (y or x): W adjacent z positions, line element i at
// o * s_outer + c + i * s_line (blockIdx.y = o, blockIdx.x * W + lane = c)
template <class T, int L, int E, int W, bool FX = false>
__global__ void __launch_bounds__(W *(L / E), min_blocks3(W *(L / E))) k3_col(Pass3Args a)
{
    pdl_wait();
    using C = cplx_t<T>;
    constexpr int TM = Plan<L, E>::TL;
    constexpr int NT = W * TM;
    extern __shared__ __align__(16) unsigned char smraw[];
    __shared__ double red[32];
    C *sm = reinterpret_cast<C *>(smraw);
    const int tid = threadIdx.x;
    const int c = tid % W, t = tid / W;
    const size_t base = (size_t)blockIdx.y * a.s_outer + (size_t)blockIdx.x * W + c + (size_t)t * a.s_line;
    const size_t stride = (size_t)TM * a.s_line;
    constexpr ColPad CP = col_pad(sizeof(C), L, W, E);
    const ColLayout<W, CP.sh, CP.p> lay{c};
    const CtaBarrier bar{};
    C *psi = static_cast<C *>(a.psi);
    const stw_t<C> *tw = static_cast<const stw_t<C> *>(a.tw);

    C x[E];
#pragma unroll
    for (int e = 0; e < E; ++e) x[e] = ld_stream(psi + base + e * stride);
    if (a.kinetic) {
        line_fft<C, L, E, false>(x, sm, lay, bar, t, tw);
        double s1 = 0, s0 = 0;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            const int k = t + e * TM;
            const double f = (double)(k > L / 2 ? L - k : k);
            const double m = abs2d(x[e]);
            s1 += m * f * f;
            s0 += m;
        }
        s1 = block_sum<NT>(s1, red);
        s0 = block_sum<NT>(s0, red);
        if (tid == 0) {
            const size_t cta = (size_t)blockIdx.y * gridDim.x + blockIdx.x;
            a.partials[2 * cta] = s1;
            a.partials[2 * cta + 1] = s0;
        }
        return;
    }
    axis_ops<C, L, E, FX>(x, sm, lay, bar, t, tw, a, [=](int e) { return base + e * stride; });
    C *o = const_cast<C *>(opaque(psi));
#pragma unroll
    for (int e = 0; e < E; ++e) st_stream(o + base + e * stride, x[e]);
}

}  // namespace qsg
