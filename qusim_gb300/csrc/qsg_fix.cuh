// qsg_fix.cuh -- complex128 line transforms in 64-bit block fixed point.
//
// GB300 runs FP64 at 2 instructions per clock and SM (measured: dfma 2.0,
// dadd 1.7, conversions to and from double 2.0), but 64-bit integer adds at 59
// and 32 x 32 + 64 multiply-adds (IMAD.WIDE) at 25-32.  A transform is mostly
// additions, so complex128 lines are transformed on integers: the line's values
// become v * 2^ex with one exponent per line (per tile for column tiles), the
// butterflies add 64-bit integers exactly, the twiddle products round to the
// last place, and the line goes back to double at the end.
//
// Precision.  Before a product the largest component of a line is between 2^57
// and 2^61 units (re-scaled after a stage by the largest magnitude the stage left,
// a reduction that rides on the exchange's barrier).  A product divides by four
// and is off by at most one unit of its result (half a unit of rounding, half of
// the low words' product left out), so by at most 2^-55 of the line's largest
// component, and by 2^-56.7 rms where that sits at 2^57 (2^-60.7 at 2^61).  Two
// products in a row keep that bound: the first one does not divide (mul_full).
// Taking a line up from doubles rounds to nearest, at 2^-59 of its largest
// component.  A double's rounding is 2^-53 of each value; a small component of a
// line has fewer significant bits here, but an FFT's error is relative to the
// line's norm in either arithmetic.
// A unit-modulus factor w is stored as {re hi, re lo, im hi, im lo}: hi =
// round(w 2^30), lo = the rest at 2^-62, so w is held to 2^-63.
#pragma once

namespace qsg {

struct Fix {
    long long x, y;
};
// table entry of a unit-modulus factor: {re hi, re lo, im hi, im lo}
using fixw = int4;

template <> struct RealOf<Fix> { using type = long long; };

__device__ __forceinline__ int fix_hi(long long v) { return (int)(v >> 32); }
__device__ __forceinline__ int fix_lo(long long v) { return (int)v; }
// v = fix_hir(v) 2^32 + (signed) fix_lo(v): the high word rounded up where the low word, taken as signed, is negative
__device__ __forceinline__ int fix_hir(long long v) { return fix_hi(v) + (int)((unsigned)fix_lo(v) >> 31); }
// c + a b in 64 bits (IMAD.WIDE)
__device__ __forceinline__ long long fix_mad(int a, int b, long long c) { return (long long)a * b + c; }

// v / 2^r, rounded to nearest, halves to even (r = 1, 2: a fixed direction would
// be a drift of an eighth to a quarter of a unit per rounding)
__device__ __forceinline__ long long fix_shr(long long v, int r)
{
    return (v + ((1 << (r - 1)) - 1 + ((fix_lo(v) >> r) & 1))) >> r;
}

// a w / 4 for |a.x|, |a.y| < 2^61.  With a = h 2^32 + l and w = wh 2^-30 + wl 2^-62,
// a w / 4 = h wh + (h wl + l wh) 2^-32 (+ l wl 2^-64, left out: below half a unit);
// the middle sum is rounded (the 2^31).  The product with an exact 1, -1, i or -i
// ends on a half a quarter of the time, and all of these rounding up would be a
// drift (at every site where V = 0, and in each stage's first butterfly).  EVEN
// rounds those of a 1 to even, at two instructions per component; the stage
// twiddles' tables hold the zero part of such a factor as 2^-62 instead
// (put_twiddle), so that the sign of the other component decides.
template <bool EVEN = false> __device__ __forceinline__ Fix fix_twmul(Fix a, fixw w)
{
    const int xh = fix_hir(a.x), xl = fix_lo(a.x), yh = fix_hir(a.y), yl = fix_lo(a.y);
    const int nh = -w.z, nl = -w.w;
    const long long cr = EVEN ? 0x7fffffffu + (xl & 4) : 0x80000000u, ci = EVEN ? 0x7fffffffu + (yl & 4) : 0x80000000u;
    long long tr = fix_mad(xh, w.y, cr), ti = fix_mad(xh, w.w, ci);
    tr = fix_mad(xl, w.x, tr);
    ti = fix_mad(xl, w.z, ti);
    tr = fix_mad(yh, nl, tr);
    ti = fix_mad(yh, w.y, ti);
    tr = fix_mad(yl, nh, tr);
    ti = fix_mad(yl, w.x, ti);
    Fix r;
    r.x = fix_mad(yh, nh, fix_mad(xh, w.x, tr >> 32));
    r.y = fix_mad(yh, w.x, fix_mad(xh, w.z, ti >> 32));
    return r;
}

// a w for |a| < 2^61.5: fix_twmul's sums in units four times as fine, with the low
// words' product, to half a unit
__device__ __forceinline__ Fix fix_twmul_full(Fix a, fixw w)
{
    const int xh = fix_hir(a.x), xl = fix_lo(a.x), yh = fix_hir(a.y), yl = fix_lo(a.y);
    const int nh = -w.z, nl = -w.w;
    long long tr = fix_mad(xh, w.y, (1ll << 29) + __mulhi(xl, w.y));
    long long ti = fix_mad(xh, w.w, (1ll << 29) + __mulhi(xl, w.w));
    tr = fix_mad(xl, w.x, tr);
    ti = fix_mad(xl, w.z, ti);
    tr = fix_mad(yh, nl, tr + __mulhi(yl, nl));
    ti = fix_mad(yh, w.y, ti + __mulhi(yl, w.y));
    tr = fix_mad(yl, nh, tr);
    ti = fix_mad(yl, w.x, ti);
    Fix r;
    r.x = fix_mad(yh, nh, fix_mad(xh, w.x, 0)) * 4 + (tr >> 30);
    r.y = fix_mad(yh, w.x, fix_mad(xh, w.z, 0)) * 4 + (ti >> 30);
    return r;
}

// u / sqrt(2), to one unit
__device__ __forceinline__ long long fix_h(long long u)
{
    constexpr int HH = 1518500250, HL = -51432894;  // 2^31 / sqrt(2) = HH + HL 2^-32
    const int h = fix_hir(u), l = fix_lo(u);
    const long long t = fix_mad(l, HH, fix_mad(h, HL, 1ll << 31));
    const long long a = fix_mad(h, HH, t >> 32);
    return a + a;
}

template <> struct Roots<Fix> {
    template <bool INV> static __device__ __forceinline__ Fix w8_1(Fix a)
    {
        return INV ? Fix{fix_h(a.x - a.y), fix_h(a.x + a.y)} : Fix{fix_h(a.x + a.y), fix_h(a.y - a.x)};
    }
    template <bool INV> static __device__ __forceinline__ Fix w8_3(Fix a)
    {
        return INV ? Fix{-fix_h(a.x + a.y), fix_h(a.x - a.y)} : Fix{fix_h(a.y - a.x), -fix_h(a.x + a.y)};
    }
};
template <> struct RootsOf<Fix, fixw> { using type = Roots<Fix>; };

// OR of the magnitudes' high words over a thread's slots (its bit length bounds every component's)
template <int E> __device__ __forceinline__ unsigned fix_or(const Fix (&v)[E])
{
    unsigned m = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const int a = fix_hi(v[e].x), b = fix_hi(v[e].y);
        m |= (unsigned)(a ^ (a >> 31));
        m |= (unsigned)(b ^ (b >> 31));
    }
    return m;
}

// Reduction over the threads that share a layout's exponent (a line of TL
// threads; a column tile: the CTA).  Lines within a warp shuffle; larger groups
// OR / MAX one word per warp into the padding words of their exchange buffer.
// `put` runs before a barrier of the group, `get` after it.  OP 0: OR, 1: max.
template <int TL, class Lay, int OP> struct FixReduce {
    static constexpr bool WARP = !Lay::kTile && TL <= 32;
    static __device__ __forceinline__ unsigned op(unsigned a, unsigned b) { return OP ? (a > b ? a : b) : (a | b); }
    static __device__ __forceinline__ unsigned put(unsigned v, unsigned *word)
    {
        if constexpr (WARP) {
            const unsigned lane = threadIdx.x & 31;
            const unsigned mask = TL == 32 ? 0xffffffffu : ((1u << (TL & 31)) - 1u) << (lane & ~(unsigned)(TL - 1));
#pragma unroll
            for (int o = TL / 2; o > 0; o >>= 1) v = op(v, __shfl_xor_sync(mask, v, o));
            return v;
        } else {
            v = OP ? __reduce_max_sync(0xffffffffu, v) : __reduce_or_sync(0xffffffffu, v);
            if ((threadIdx.x & 31) == 0) {
                if (OP)
                    atomicMax(word, v);
                else
                    atomicOr(word, v);
            }
            return v;
        }
    }
    static __device__ __forceinline__ unsigned get(unsigned v, const unsigned *word)
    {
        return WARP ? v : *const_cast<const volatile unsigned *>(word);
    }
};

// the double d as units of 2^(emax - 1023 - 52 - UP): its 53-bit significand from bit 52 + UP
// down, shifted by the distance of its exponent from emax and rounded to nearest
template <int UP = 6> __device__ __forceinline__ long long fix_from(double d, int emax)
{
    const int hi = __double2hiint(d);
    const unsigned lo = (unsigned)__double2loint(d);
    const int e = (hi >> 20) & 0x7ff;
    const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
    int sh = emax - e;
    sh = sh > 63 ? 63 : sh;
    const unsigned long long m = (((unsigned long long)mh << 32 | lo) << (UP + 1)) >> sh;
    const long long s = (long long)(hi >> 31);
    if constexpr (UP < 10) return (((long long)m ^ s) + 1) >> 1;  // -((m + 1) / 2) = (~m + 1) >> 1
    return ((long long)((m + 1) >> 1) ^ s) - s;                    // (all 64 bits of m in use)
}

// v 2^ex as a double, rounded to nearest (halves away from zero); ex keeps every result in the normal range (see fix_out)
__device__ __forceinline__ double fix_to(long long v, int ex)
{
    const int s = fix_hi(v) >> 31;
    const long long sl = s;
    const unsigned long long a = (unsigned long long)((v ^ sl) - sl);
    const unsigned ah = (unsigned)(a >> 32), al = (unsigned)a;
    const int lz = __clz(ah ? (int)ah : (int)al) + (ah ? 0 : 32);  // 1 .. 64
    const unsigned long long m = ((a << (lz - 1)) + 0x200ull) >> 10;  // the leading one at bit 52 (53 on a carry)
    // biased exponent - 1: the leading one adds the 1 (and a carry one more)
    const int eb = a ? ex + (63 - lz) + 1022 : 0;
    return __hiloint2double((int)(((unsigned)(m >> 32) + ((unsigned)eb << 20)) | ((unsigned)s & 0x80000000u)),
                            (int)(unsigned)m);
}

// double line -> fixed point; returns the exponent (value = v 2^ex), and whether the line is finite.
// mx: the largest high word (sign cleared) of the line.  A line near the bottom of the range
// is scaled by an exact power of two first, which also makes its subnormal values normal.
template <int E> __device__ __forceinline__ int fix_in(double2 (&x)[E], Fix (&v)[E], unsigned mx, bool *finite)
{
    int emax = (int)(mx >> 20), up = 0;
    *finite = emax != 0x7ff;
    if (emax < 64) {
        up = 200;
        emax += up;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            x[e].x *= 0x1p200;
            x[e].y *= 0x1p200;
        }
    }
#pragma unroll
    for (int e = 0; e < E; ++e) {
        v[e].x = fix_from(x[e].x, emax);
        v[e].y = fix_from(x[e].y, emax);
    }
    return emax - up - 1023 - 58;
}

template <int E> __device__ __forceinline__ unsigned fix_absmax(const double2 (&x)[E])
{
    unsigned m = 0;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        const unsigned a = (unsigned)__double2hiint(x[e].x) & 0x7fffffffu, b = (unsigned)__double2hiint(x[e].y) & 0x7fffffffu;
        m = a > m ? a : m;
        m = b > m ? b : m;
    }
    return m;
}

// fixed point -> double.  Exponents whose results could leave the normal range
// go through a second, exact power of two; a line that held an infinity or a NaN
// becomes NaN throughout, as its transform is.
template <int E> __device__ __forceinline__ void fix_out(const Fix (&v)[E], double2 (&x)[E], int ex, bool finite)
{
    const bool tiny = ex < -900, huge = ex > 900;
    const int e2 = tiny ? ex + 400 : huge ? ex - 400 : ex;
#pragma unroll
    for (int e = 0; e < E; ++e) {
        x[e].x = fix_to(v[e].x, e2);
        x[e].y = fix_to(v[e].y, e2);
    }
    if (tiny || huge || !finite) {
        const double sc = !finite ? __hiloint2double(0x7ff80000, 0) : tiny ? 0x1p-400 : 0x1p400;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            x[e].x *= sc;
            x[e].y *= sc;
        }
    }
}

// Scale a line so that every component is below 2^61 units and the largest is
// not far below: m is the OR of the magnitudes' high words.
template <int E> __device__ __forceinline__ void fix_norm(Fix (&v)[E], unsigned m, int &ex)
{
    const int top = 31 - __clz((int)m);  // bit length - 1 of the high words (-1: all below 2^32)
    if (top > 28) {
        const int r = top - 28;  // 1 or 2
#pragma unroll
        for (int e = 0; e < E; ++e) {
            v[e].x = fix_shr(v[e].x, r);
            v[e].y = fix_shr(v[e].y, r);
        }
        ex += r;
    } else if (top < 25) {
        const int l = 28 - top;
#pragma unroll
        for (int e = 0; e < E; ++e) {
            v[e].x <<= l;
            v[e].y <<= l;
        }
        ex -= l;
    }
}

// A phase table of fixed-point factors ends in a flag entry, not zero when a
// factor was not finite (an infinite potential): such a table makes every line
// it multiplies NaN, as the factor itself would after the next transform.
__device__ __forceinline__ bool fix_flagged(const fixw *entry) { return __ldg(&entry->x) != 0; }

// A complex128 line held in fixed point by its threads: slot e of thread t is
// element t + e L / E, as in the register lines of qsg_fft.cuh, with value
// v 2^ex.  Transforms and unit-modulus products chain without going back to
// double.  Magnitudes (of the complex values, in units): a transform takes
// |v| <= 2^59.5 and leaves |v| < 2^63 / sqrt(2); scale() brings components
// below 2^61; a product takes that and leaves |v| <= 2^59.5; mul_full takes and
// leaves |v| <= 2^61.5, so another product follows it, or the line's end.
//
// Reductions beyond one warp go through four words in the padding of the
// exchange buffer: word 0 for load(), words 1 .. 3 in turn for the others.  A
// reduction's word is zeroed before the barrier of the reduction before it,
// when the word's last readers (three reductions back) are behind a barrier.
template <int L, int E> struct FixLine {
    Fix v[E];
    int ex;
    int r;        // next reduction's word
    bool finite;  // false: the line holds an infinity or a NaN, and so do all its results

    template <class Lay> static __device__ __forceinline__ unsigned *words(double2 *smd, const Lay &lay)
    {
        return reinterpret_cast<unsigned *>(smd + lay.pad_slot());
    }
    // double line -> fixed point.  x is the line (changed where it is tiny).
    template <class Lay, class Bar>
    __device__ __forceinline__ void load(double2 (&x)[E], double2 *smd, const Lay &lay, const Bar &bar, int t)
    {
        static_assert(sizeof(Fix) == sizeof(double2), "the exchange buffer is shared");
        using Red = FixReduce<L / E, Lay, 1>;
        unsigned *w = words(smd, lay);
        unsigned mx = fix_absmax(x);
        if constexpr (Red::WARP) {
            mx = Red::put(mx, w);
        } else {
            // word 0's last readers are behind a later barrier; the others' may still be
            // reading until every thread is here
            if (lay.leader(t)) w[0] = 0;
            bar();
            Red::put(mx, w);
            if (lay.leader(t)) w[1] = 0;
            bar();
            mx = Red::get(mx, w);
        }
        r = 1;
        ex = fix_in(x, v, mx, &finite);
    }
    __device__ __forceinline__ void store(double2 (&x)[E]) const { fix_out(v, x, ex, finite); }
    __device__ __forceinline__ void conj()
    {
#pragma unroll
        for (int e = 0; e < E; ++e) v[e].y = -v[e].y;
    }
    __device__ __forceinline__ static int after(int i) { return i == 3 ? 1 : i + 1; }

    // components below 2^61, the largest not far below (after a transform, before a product)
    template <class Lay, class Bar>
    __device__ __forceinline__ void scale(double2 *smd, const Lay &lay, const Bar &bar, int t)
    {
        using Red = FixReduce<L / E, Lay, 0>;
        unsigned *w = words(smd, lay);
        const unsigned m = Red::put(fix_or(v), w + r);
        if constexpr (!Red::WARP) {
            if (lay.leader(t)) w[after(r)] = 0;
            bar();
        }
        fix_norm(v, Red::get(m, w + r), ex);
        if constexpr (!Red::WARP) r = after(r);
    }
    // v *= f(e); H < E: only the first H slots (the others are not used afterwards).  mul_v: of a
    // potential table, whose factors may be 1 over most of the line
    template <int H = E, bool EVEN = false, class F> __device__ __forceinline__ void mul(F f)
    {
#pragma unroll
        for (int e = 0; e < H; ++e) v[e] = fix_twmul<EVEN>(v[e], f(e));
        ex += 2;
    }
    template <int H = E, class F> __device__ __forceinline__ void mul_v(F f) { mul<H, true>(f); }
    // the same without the division by four: before another product
    template <class F> __device__ __forceinline__ void mul_full(F f)
    {
#pragma unroll
        for (int e = 0; e < E; ++e) v[e] = fix_twmul_full(v[e], f(e));
    }
    // The end of a step: the line rounded to doubles and taken up again, as a call that ended
    // here would store it and the next one load it (H < E: slots from H on zero).  A step split
    // across calls, chunks of the server or reads of the state then equals one call bit for bit.
    template <int H = E, class Lay, class Bar>
    __device__ __forceinline__ void round(double2 (&x)[E], double2 *smd, const Lay &lay, const Bar &bar, int t)
    {
        const bool ok = finite;
        store(x);
#pragma unroll
        for (int e = H; e < E; ++e) x[e] = double2{0, 0};
        load(x, smd, lay, bar, t);
        finite = finite && ok;
    }
    // the product's change of scale without a product
    __device__ __forceinline__ void quarter()
    {
#pragma unroll
        for (int e = 0; e < E; ++e) {
            v[e].x = fix_shr(v[e].x, 2);
            v[e].y = fix_shr(v[e].y, 2);
        }
        ex += 2;
    }

    // one Stockham stage (fft_stage's data movement)
    template <int S, class Lay, class Bar>
    __device__ __forceinline__ void stage(double2 *smd, const Lay &lay, const Bar &bar, int t, const fixw *__restrict__ tw)
    {
        using P = Plan<L, E>;
        constexpr int RL = P::radix_log(S);
        constexpr int R = 1 << RL;
        static_assert(R <= 8, "radix 2, 4 or 8: a radix-8 sum grows by at most 8");
        constexpr int PL = P::p_log(S);
        constexpr int PP = 1 << PL;
        constexpr int J = E / R;
        constexpr int TL = P::TL;
        constexpr int TWO = P::tw_offset(S);
#pragma unroll
        for (int j = 0; j < J; ++j) {
            Fix u[R];
#pragma unroll
            for (int q = 0; q < R; ++q) u[q] = v[j + q * J];
            if constexpr (PP > 1) {
                const int k = (t + j * TL) & (PP - 1);
                u[0].x = fix_shr(u[0].x, 2);
                u[0].y = fix_shr(u[0].y, 2);
#pragma unroll
                for (int q = 1; q < R; ++q) u[q] = fix_twmul(u[q], __ldg(&tw[TWO + (q - 1) * PP + k]));
            }
            dft<R, false, Fix, fixw>(u);
#pragma unroll
            for (int q = 0; q < R; ++q) v[j + q * J] = u[q];
        }
        if constexpr (PP > 1) ex += 2;
        if constexpr (S + 1 < P::NST) {
            Fix *sm = reinterpret_cast<Fix *>(smd);
            using Red = FixReduce<TL, Lay, 0>;
            unsigned *w = words(smd, lay);
            const unsigned m = Red::put(fix_or(v), w + r);
            bar();  // every reader of the previous stage is done with the buffer
            if constexpr (!Red::WARP) {
                if (lay.leader(t)) w[after(r)] = 0;
            }
#pragma unroll
            for (int j = 0; j < J; ++j) {
                const int b = t + j * TL;
                const int k = b & (PP - 1);
                const int o = ((b - k) << RL) + k;
#pragma unroll
                for (int q = 0; q < R; ++q) sm[lay(o + q * PP)] = v[j + q * J];
            }
            bar();
#pragma unroll
            for (int e = 0; e < E; ++e) v[e] = sm[lay(t + e * TL)];
            fix_norm(v, Red::get(m, w + r), ex);
            if constexpr (!Red::WARP) r = after(r);
        }
    }
    template <int S = 0, class Lay, class Bar>
    __device__ __forceinline__ void fft(double2 *smd, const Lay &lay, const Bar &bar, int t, const fixw *__restrict__ tw)
    {
        if constexpr (S < Plan<L, E>::NST) {
            stage<S>(smd, lay, bar, t, tw);
            fft<S + 1>(smd, lay, bar, t, tw);
        }
    }
};

// Forward transform of a complex128 line (line_fft's contract).
// Per step against FP64 butterflies and products, with the chained passes and the
// plans that came with them: 1024^2 O4 1026 -> 235 us, a 1000-site wall 593 -> 122,
// a 131072-site line (O2) 79.8 -> 25.8, 450 x 700 1991 -> 438.
template <int L, int E, class Lay, class Bar>
__device__ __forceinline__ void line_fft_fix(double2 (&x)[E], double2 *smd, const Lay &lay, const Bar &bar, int t,
                                             const fixw *__restrict__ tw)
{
    FixLine<L, E> f;
    f.load(x, smd, lay, bar, t);
    f.fft(smd, lay, bar, t, tw);
    f.store(x);
}

}  // namespace qsg
