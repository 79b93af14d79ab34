// wlc_fixfft.cuh -- the line FFTs of the FP64 form in 64-bit block floating
// point.
//
// Why: the FP64 pipe of sm_103a issues 2 lane operations per clock and SM
// (measured 1.67 at a 2.07 GHz nominal clock, DADD and DFMA alike, 64 clocks
// latency), its integer ALUs 64 64-bit adds (measured 59) and about 14 signed
// 32x32+64 multiply-adds.  A radix butterfly is mostly additions, so it runs
// about seven times faster on 64-bit integers than on doubles.
//
// Form: the R complex numbers of one register butterfly share an exponent E,
// value = v 2^(E - 1023 - kTop), with the largest component's leading bit at
// kTop = 56.  Four bits stay below the 53-bit significand of the largest
// component, and log2(16 sqrt(2)) + 2 bits above it for the growth of a line
// and one addition after it.  Butterflies of one line meet at the largest
// exponent (right shifts by the difference).  Every input is read as the
// double it is, and what leaves a line FFT as a double is rounded once; the
// additions between are exact to 2^-56 of the line's largest value, so the
// error against 64-bit arithmetic is below that of FP64 butterflies.
// Measured at 64^3, L = 10 (M = 121), launches timed one by one: pass A 1.42 ->
// 0.65 ms, pass C 1.23 -> 0.37 ms (0.53 and 0.34 with launch shapes by size), the two z-FFTs of pass B 0.6 ms less; one
// step's error against 80-bit arithmetic 5.3e-16 -> 4.5e-16 of the result's
// norm (1.50e-15 -> 1.45e-15 at the worst point).
// Not-a-number and infinite inputs, and a correction in floats that has
// overflowed, turn all outputs of their line into NaN.  Numbers keep their
// bits down to the smallest subnormal; results below 2^-920 or above 2^977 are
// rounded by the library's ldexp.
#pragma once
#include <cstdint>

#include "wlc_fft.cuh"

namespace wlc {

constexpr int kTop = 56;       // bit of the largest component after normalisation
constexpr int kExpLow = 64;     // shared (biased) exponents below are tiny numbers: d2fx_low, lift_tiny
constexpr int kLift = 512;
constexpr int kExpMin = -100;   // below every shared exponent
constexpr int kExpBad = 20000;  // exponent of a line with non-finite input

// a fixed-point number; as a constant it holds value * 2^62
struct fx {
    long long v;
    fx() = default;
    __host__ __device__ constexpr explicit fx(double c) : v((long long)(c * 4611686018427387904.0)) {}
};
__device__ __forceinline__ fx mkfx(long long v) {
    fx r;
    r.v = v;
    return r;
}
__device__ __forceinline__ fx operator+(fx a, fx b) { return mkfx(a.v + b.v); }
__device__ __forceinline__ fx operator-(fx a, fx b) { return mkfx(a.v - b.v); }
__device__ __forceinline__ fx operator-(fx a) { return mkfx(-a.v); }
__device__ __forceinline__ fx operator*(int sign, fx a) { return sign > 0 ? a : -a; }  // sign = +-1

// halves of a factor, v = h 2^32 + l with both signed (every partial product
// is a signed 32 x 32 -> 64 multiply-add; the product of the two low halves
// is left out)
struct fxh {
    int h, l;
};
__device__ __forceinline__ fxh halves(long long v) {
    return {(int)(v >> 32) + (int)((unsigned)v >> 31), (int)(unsigned)v};
}
__device__ __forceinline__ long long join_halves(fxh a) { return ((long long)a.h << 32) + a.l; }
// hi*2^64 + mid*2^32 -> units of 2^62 (the product with a constant of 62
// fraction bits); the middle sums start from kHalf, so that the shift rounds
constexpr long long kHalf = 1LL << 29;
__device__ __forceinline__ long long fx_join(long long hi, long long mid) { return (hi << 2) + (mid >> 30); }
__device__ __forceinline__ fx operator*(fx a, fx b) {
    const fxh x = halves(a.v), y = halves(b.v);
    return mkfx(fx_join((long long)x.h * y.h, (long long)x.h * y.l + ((long long)x.l * y.h + kHalf)));
}

struct __align__(16) fxc {
    fx x, y;
};
// twiddle factor, split into halves once per CTA
struct __align__(16) fxw {
    fxh x, y;
};
__device__ __forceinline__ fxw make_fxw(double2 w) {
    fxw r;
    r.x = halves(__double2ll_rn(w.x * 4611686018427387904.0));
    r.y = halves(__double2ll_rn(w.y * 4611686018427387904.0));
    return r;
}
// a * w (DIR < 0) or a * conj(w): the two products of a component share one join
template <int DIR> __device__ __forceinline__ fxc fx_twiddle(fxc a, const fxw& w) {
    const fxh x = halves(a.x.v), y = halves(a.y.v);
    // x w.x -+ y w.y and x w.y +- y w.x
    const long long h1 = (long long)x.h * w.x.h, m1 = (long long)x.h * w.x.l + ((long long)x.l * w.x.h + kHalf);
    const long long h2 = (long long)y.h * w.y.h, m2 = (long long)y.h * w.y.l + ((long long)y.l * w.y.h + kHalf);
    const long long h3 = (long long)x.h * w.y.h, m3 = (long long)x.h * w.y.l + ((long long)x.l * w.y.h + kHalf);
    const long long h4 = (long long)y.h * w.x.h, m4 = (long long)y.h * w.x.l + ((long long)y.l * w.x.h + kHalf);
    fxc r;
    if (DIR < 0) {
        r.x.v = ((h1 - h2) << 2) + ((m1 >> 30) - (m2 >> 30));
        r.y.v = ((h3 + h4) << 2) + ((m3 >> 30) + (m4 >> 30));
    } else {
        r.x.v = ((h1 + h2) << 2) + ((m1 >> 30) + (m2 >> 30));
        r.y.v = ((h4 - h3) << 2) + ((m4 >> 30) - (m3 >> 30));
    }
    return r;
}

// ---------------------------------------------------------- conversions
__device__ __forceinline__ int dexp(double d) { return (__double2hiint(d) >> 20) & 0x7ff; }
__device__ __forceinline__ unsigned long long shr_u64(unsigned long long v, int s) {  // 0 for s >= 64
    unsigned long long r;
    asm("shr.u64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
}
__device__ __forceinline__ long long sar_s64(long long v, int s) {  // sign for s >= 64
    long long r;
    asm("shr.s64 %0, %1, %2;" : "=l"(r) : "l"(v), "r"(s));
    return r;
}
// v / 2^s to the nearest, s >= 1 (halves up; 0 or so for s > 64)
__device__ __forceinline__ long long round_shift(long long v, int s) { return (sar_s64(v, s - 1) + 1) >> 1; }
// d as a fixed-point number under exponent E >= d's own (E's leading bit at
// TOP), E >= kExpLow (a zero or subnormal d then counts as zero)
template <int TOP = kTop> __device__ __forceinline__ fx d2fx(double d, int E) {
    const int hi = __double2hiint(d), lo = __double2loint(d);
    const int s = E - ((hi >> 20) & 0x7ff);
    const unsigned mh = ((unsigned)hi & 0xfffffu) | 0x100000u;
    const unsigned long long m = (((unsigned long long)mh << 32) | (unsigned)lo) << (TOP - 51);
    const long long v = (long long)((shr_u64(m, s) + 1) >> 1);
    const long long sg = (long long)(hi >> 31);
    return mkfx((v ^ sg) - sg);
}
// the same under any E >= 1, for subnormal d as well
__device__ __forceinline__ fx d2fx_low(double d, int E) {
    const long long b = __double_as_longlong(d);
    const int e = dexp(d);
    const unsigned long long m = ((b & 0xfffffffffffffll) | (e ? 1ll << 52 : 0ll)) << (kTop - 51);
    const long long v = (long long)((shr_u64(m, E - max(e, 1)) + 1) >> 1);
    return mkfx(b < 0 ? -v : v);
}
// value of v under an exponent for which fx2d and fx2d_cvt do not hold
__device__ __forceinline__ bool fx_rare(int E) { return (unsigned)(E - 100) >= 1900u; }
static __device__ __noinline__ double fx2d_rare(long long v, int E) {
    if (E >= kExpBad / 2) return __longlong_as_double(0x7ff8000000000000LL);
    return v == 0 ? 0.0 : ldexp((double)v, E - 1023 - kTop);
}
// the doubles v[j * step], j < n, times 2^kLift (exact); returns the largest
// exponent field then, 0 if all are zero
static __device__ __noinline__ int lift_tiny(double* v, int step, int n) {
    int E = 0;
#pragma unroll 1
    for (int j = 0; j < n; ++j) {
        const double x = v[j * step] * 0x1p512;
        v[j * step] = x;
        E = max(E, dexp(x));
    }
    return E;
}
// d as a float, round to nearest even, on the integer ALUs (the conversion
// instruction runs on the FP64 pipe; only zeros and what becomes a subnormal
// float go there)
__device__ __forceinline__ float d2f(double d) {
    const long long b = __double_as_longlong(d);
    const long long r = b + 0x0fffffff + ((b >> 29) & 1);
    const int e = (int)((r >> 52) & 0x7ff) - (1023 - 127);
    const unsigned m = (unsigned)(r >> 29) & 0x7fffffu, sg = (unsigned)(b >> 32) & 0x80000000u;
    float f = __uint_as_float(e >= 255 ? sg | 0x7f800000u | ((unsigned long long)b << 1 > 0x7ffull << 53 ? 1u : 0u)
                                       : sg | ((unsigned)e << 23) | m);
    asm("{ .reg .pred p; setp.le.s32 p, %2, 0; @p cvt.rn.f32.f64 %0, %1; }" : "+f"(f) : "d"(d), "r"(e));
    return f;
}
// v under exponent E as a double by the conversion instruction: fewer
// instructions than fx2d, on the FP64 pipe (for loops whose other work is on
// the integer ALUs)
__device__ __forceinline__ double fx2d_cvt(long long v, int E) {
    const double d = __ll2double_rn(v);
    return v == 0 ? 0.0 : __hiloint2double(__double2hiint(d) + ((E - 1023 - kTop) << 20), __double2loint(d));
}
// value of v under exponent E as a double (round to nearest, halves to even)
__device__ __forceinline__ double fx2d(fx q, int E) {
    const long long sg = q.v >> 63;
    const unsigned long long a = (unsigned long long)((q.v ^ sg) - sg);
    const int n = __clzll((long long)a);
    const unsigned long long m = a << ((n - 1) & 63);
    const unsigned long long r = (m + 0x1ffull + ((m >> 10) & 1ull)) >> 10;  // 53 bits, leading one at bit 52
    const int e = E + (62 - kTop) - n;  // the leading one adds the last unit of the exponent
    long long b = (long long)r + ((long long)e << 52);
    b |= sg & (long long)0x8000000000000000ull;
    return a == 0 ? 0.0 : __longlong_as_double(b);
}

// E of R complex doubles
template <int R> __device__ __forceinline__ int shared_exp(const double2* d) {
    int E = 0;
#pragma unroll
    for (int n = 0; n < R; ++n) E = max(E, max(dexp(d[n].x), dexp(d[n].y)));
    return E == 2047 ? kExpBad : E;
}
// R complex numbers with exponents e[n] brought to one exponent under which
// the largest component's leading bit is at kTop; returns that exponent
template <int R> __device__ __forceinline__ int renormalise(fxc* v, const int* e) {
    int top = kExpMin + kTop;
#pragma unroll
    for (int n = 0; n < R; ++n) {
        const long long m = (v[n].x.v ^ (v[n].x.v >> 63)) | (v[n].y.v ^ (v[n].y.v >> 63));
        top = max(top, e[n] + 63 - __clzll(m));
    }
    const int E = top - kTop;
#pragma unroll
    for (int n = 0; n < R; ++n) {
        const int s = E - e[n], l = max(1 - s, 0), r = max(s - 1, 0);  // s = r + 1 - l
        v[n].x.v = (sar_s64(v[n].x.v << l, r) + 1) >> 1;
        v[n].y.v = (sar_s64(v[n].y.v << l, r) + 1) >> 1;
    }
    return E;
}

// ---------------------------------------------------------- line FFTs
// bits dropped before the second sub-pass so that a whole line stays below
// 2^(kTop + 1) * 16 sqrt(2)
template <int N> __host__ __device__ constexpr int fx_drop() {
    int b = 1;
    while ((16 << b) < N) ++b;
    return b;
}
// exponents kept between the two sub-passes of a batch of lines
template <int N> __host__ __device__ constexpr int fx_exps(int nlines) {
    return Plan<N>::N2 == 1 ? 0 : nlines * (Plan<N>::N1 > Plan<N>::N2 ? Plan<N>::N1 : Plan<N>::N2);
}

// a float as a fixed-point number under exponent E >= fexp of the largest |f|'s
// bits.  fexp of zero: 0 (a correction that vanishes must not raise its line's
// exponent); of an infinity or not-a-number: kExpBad
__device__ __forceinline__ int fexp(int u) {
    return u >= 0x7f800000 ? kExpBad : u == 0 ? 0 : max(u >> 23, 1) + (1023 - 127);
}
__device__ __forceinline__ fx f2fx(float f, int E) {
    const int u = __float_as_int(f), e = (u >> 23) & 0xff;
    const long long m = (long long)((u & 0x7fffff) | (e ? 0x800000 : 0)) << (kTop - 22);
    const long long v = round_shift(m, E - (max(e, 1) + 1023 - 127) + 1);
    return mkfx(u < 0 ? -v : v);
}

// Input of a line FFT: doubles, doubles less a correction in floats, or fixed-point numbers with an exponent per
// (line, element).
struct FromDoubles {
    static constexpr bool dbl = true, less = false;
};
struct FromDoublesLess {  // correction of (line, element) at c[line * stride + element]
    static constexpr bool dbl = true, less = true;
    const float2* c;
    int stride;
};
template <typename F> struct FromFixed {
    static constexpr bool dbl = false;
    F f;
    __device__ int operator()(int line, int elem) const { return f(line, elem); }
};
template <typename F> __device__ __forceinline__ FromFixed<F> from_fixed(F f) { return FromFixed<F>{f}; }

// the R elements base + n*step of line b into registers; returns the exponent
template <int R, typename In>
__device__ __forceinline__ int fx_load(const double2* ln, int estride, int b, int base, int step, const In& in, fxc* v) {
    if constexpr (In::dbl) {
        double2 d[R];
#pragma unroll
        for (int n = 0; n < R; ++n) d[n] = ln[(base + n * step) * estride];
        int E = shared_exp<R>(d);
        float2 c[In::less ? R : 1];
        if constexpr (In::less) {
            int u = 0;
#pragma unroll
            for (int n = 0; n < R; ++n) {
                c[n] = in.c[b * in.stride + base + n * step];
                u = max(u, max(__float_as_int(c[n].x) & 0x7fffffff, __float_as_int(c[n].y) & 0x7fffffff));
            }
            E = max(E, fexp(u));
            E = E < kExpBad ? E + 1 : E;  // room for the difference
        }
        if (E < kExpLow) {  // tiny numbers or zeros (and no correction)
            E = max(E, 1);
#pragma unroll
            for (int n = 0; n < R; ++n) {
                v[n].x = d2fx_low(d[n].x, E);
                v[n].y = d2fx_low(d[n].y, E);
            }
            return E;
        }
#pragma unroll
        for (int n = 0; n < R; ++n) {
            v[n].x = d2fx(d[n].x, E);
            v[n].y = d2fx(d[n].y, E);
            if constexpr (In::less) {
                v[n].x = v[n].x - f2fx(c[n].x, E);
                v[n].y = v[n].y - f2fx(c[n].y, E);
            }
        }
        return E;
    } else {
        int e[R];
#pragma unroll
        for (int n = 0; n < R; ++n) {
            v[n] = reinterpret_cast<const fxc*>(ln)[(base + n * step) * estride];
            e[n] = in(b, base + n * step);
        }
        return renormalise<R>(v, e);
    }
}
// the R elements base + n*step written back as doubles or fixed-point numbers
template <int R, bool OUTD>
__device__ __forceinline__ void fx_store(double2* ln, int estride, int base, int step, const fxc* v, int E) {
    if constexpr (OUTD) {
        const bool rare = fx_rare(E);
#pragma unroll
        for (int n = 0; n < R; ++n) {
            double2 d;
            if (!rare) {
                d.x = fx2d(v[n].x, E);
                d.y = fx2d(v[n].y, E);
            } else {
                d.x = fx2d_rare(v[n].x.v, E);
                d.y = fx2d_rare(v[n].y.v, E);
            }
            ln[(base + n * step) * estride] = d;
        }
    } else {
#pragma unroll
        for (int n = 0; n < R; ++n) reinterpret_cast<fxc*>(ln)[(base + n * step) * estride] = v[n];
    }
}
// R elements of the second sub-pass with their sub-transforms' exponents ex[n*estep]
template <int N, int R>
__device__ __forceinline__ int fx_meet(const double2* ln, int estride, int base, int step, const int16_t* ex, int estep,
                                       fxc* v) {
    int e[R], E = kExpMin;
#pragma unroll
    for (int n = 0; n < R; ++n) {
        v[n] = reinterpret_cast<const fxc*>(ln)[(base + n * step) * estride];
        e[n] = ex[n * estep];
        E = max(E, e[n]);
    }
#pragma unroll
    for (int n = 0; n < R; ++n) {
        const int s = E - e[n] + fx_drop<N>();
        v[n].x.v = round_shift(v[n].x.v, s);
        v[n].y.v = round_shift(v[n].y.v, s);
    }
    return E + fx_drop<N>();
}

// Batched in-place line FFTs as fft_nat2perm / fft_perm2nat (wlc_fft.cuh),
// same positions, same work split.  es: fx_exps<N>(nlines) exponents of
// scratch; el[b]: exponent of line b when the output stays fixed-point (unused
// with OUTD).
template <int N, int DIR, bool OUTD, typename In>
__device__ __forceinline__ void fx_nat2perm(double2* data, int nlines, int estride, int lstride, const fxw* tw,
                                            int16_t* es, int16_t* el, const In& in) {
    constexpr int N1 = Plan<N>::N1, N2 = Plan<N>::N2;
    if constexpr (N2 == 1) {
        for (int b = threadIdx.x; b < nlines; b += blockDim.x) {
            double2* ln = data + (size_t)b * lstride;
            fxc v[N1];
            const int E = fx_load<N1>(ln, estride, b, 0, 1, in, v);
            Dft<N1>::template run<DIR>(v);
            fx_store<N1, OUTD>(ln, estride, 0, 1, v, E);
            if (!OUTD) el[b] = (int16_t)E;
        }
        __syncthreads();
    } else {
        for (LineWalk it(nlines); it.j < N2; it.next()) {
            const int j2 = it.j;
            double2* ln = data + (size_t)it.b * lstride;
            fxc v[N1];
            const int E = fx_load<N1>(ln, estride, it.b, j2, N2, in, v);
            Dft<N1>::template run<DIR>(v);
#pragma unroll
            for (int k1 = 1; k1 < N1; ++k1)
                if (j2 != 0) v[k1] = fx_twiddle<DIR>(v[k1], tw[j2 * k1]);
            fx_store<N1, false>(ln, estride, j2, N2, v, E);
            es[it.b * N2 + j2] = (int16_t)E;
        }
        __syncthreads();
        for (LineWalk it(nlines); it.j < N1; it.next()) {
            const int k1 = it.j;
            double2* ln = data + (size_t)it.b * lstride;
            fxc v[N2];
            const int E = fx_meet<N, N2>(ln, estride, k1 * N2, 1, es + it.b * N2, 1, v);
            Dft<N2>::template run<DIR>(v);
            fx_store<N2, OUTD>(ln, estride, k1 * N2, 1, v, E);
            if (!OUTD && k1 == 0) el[it.b] = (int16_t)E;
        }
        __syncthreads();
    }
}

template <int N, int DIR, bool OUTD, typename In>
__device__ __forceinline__ void fx_perm2nat(double2* data, int nlines, int estride, int lstride, const fxw* tw,
                                            int16_t* es, int16_t* el, const In& in) {
    constexpr int N1 = Plan<N>::N1, N2 = Plan<N>::N2;
    if constexpr (N2 == 1) {
        fx_nat2perm<N, DIR, OUTD>(data, nlines, estride, lstride, tw, es, el, in);
    } else {
        for (LineWalk it(nlines); it.j < N1; it.next()) {
            const int k1 = it.j;
            double2* ln = data + (size_t)it.b * lstride;
            fxc v[N2];
            const int E = fx_load<N2>(ln, estride, it.b, k1 * N2, 1, in, v);
            Dft<N2>::template run<DIR>(v);
#pragma unroll
            for (int n2 = 1; n2 < N2; ++n2)
                if (k1 != 0) v[n2] = fx_twiddle<DIR>(v[n2], tw[n2 * k1]);
            fx_store<N2, false>(ln, estride, k1 * N2, 1, v, E);
            es[it.b * N1 + k1] = (int16_t)E;
        }
        __syncthreads();
        for (LineWalk it(nlines); it.j < N2; it.next()) {
            const int n2 = it.j;
            double2* ln = data + (size_t)it.b * lstride;
            fxc v[N1];
            const int E = fx_meet<N, N1>(ln, estride, n2, N2, es + it.b * N1, 1, v);
            Dft<N1>::template run<DIR>(v);
            fx_store<N1, OUTD>(ln, estride, n2, N2, v, E);
            if (!OUTD && n2 == 0) el[it.b] = (int16_t)E;
        }
        __syncthreads();
    }
}

}  // namespace wlc
