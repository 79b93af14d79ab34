// wlc_solve.cu -- pass B of a contour step: for one (kx, ky) column, the
// z-FFT of every harmonic coefficient, the per-wavevector solve of G(k)
// (replacing the stored dense G^-1 of Gmatrix_2dcomp_mod.f90:384-600 and
// its apply, wormlike_MDE_2dcomp_mod.f90:395-409) and the inverse z-FFT.
//
// Factorised solve (see wlc_host.cpp): G^-1 = D T^-1 D^T with
// D = Dz(alpha) Xm Dz(beta) Xp and T = A + i sigma ds |k| Rz, one
// tridiagonal system per m.  The threads of a CTA share out (kz, degree
// block) for the rotations, in registers with the generated constant
// codelets (wlc_rot_gen.cuh), and (kz, m) for the tridiagonal sweeps through
// the shared column (line stride N+1, conflict free).  Tridiagonal
// pivots come from a per-(order, block) table keyed by ix^2+iy^2+iz^2 when
// the grid spacing is isotropic.
#include <algorithm>
#include <cstdio>

#include "wlc_attr.h"
#include "wlc_fixfft.cuh"
#include "wlc_kernels.cuh"
#define WLC_ROT_TABLES
#include "wlc_rot_gen.cuh"
#include "wlc_step.h"

namespace wlc {

__device__ __forceinline__ int fold_n(int i, int n) { return i <= n / 2 ? i : i - n; }

// ---------------------------------------------------------------------
// Per-wavevector solve.  The rotations D are real matrices, so the real and
// the imaginary parts of a coefficient vector are rotated independently:
// thread (kz, part c of the complex number) works on every second word of the
// column (element i at v[i*vs], vs = 2 (N + 1) words), lanes of a warp on
// consecutive words, conflict free.  Against one thread per complex vector
// this halves the registers (the largest block, l = 12, holds 2 x 25 numbers)
// and doubles the warps of a column: FP32 pass B at 64^3, L = 10 went from 304
// to 205 us, 12 -> 24 warps an SM.
// Rotations work block by block (degree l) in registers with the generated
// constant codelets; the tridiagonal sweeps run through the shared column.

// arithmetic of the rotation codelets on plain numbers
template <typename T> struct RotReal {
    using in = T;
    using out = T;
    __device__ __forceinline__ static T mul(double c, T v) { return (T)c * v; }
    __device__ __forceinline__ static T mad(T s, double c, T v) { return fma((T)c, v, s); }
    __device__ __forceinline__ static T done(T s) { return s; }
};

// Dz(sgn * gamma) on the (m, -m) pairs of register block a (index m+l)
template <int l, typename T>
__device__ __forceinline__ void dz_block(T* a, const T* cs, int sgn) {
#pragma unroll
    for (int m = 1; m <= l; ++m) {
        const T cm = cs[2 * m], sm = sgn > 0 ? cs[2 * m + 1] : -cs[2 * m + 1];
        const T x = a[l + m], y = a[l - m];
        a[l + m] = cm * x - sm * y;
        a[l - m] = sm * x + cm * y;
    }
}

// Dz(sgn * beta) on block a, with cos/sin(m beta) generated by the
// recurrence from (cb, sb) = (cos beta, sin beta) as the block goes (no
// table held in registers across blocks)
template <int l, typename T>
__device__ __forceinline__ void dz_block_rec(T* a, T cb, T sb, int sgn) {
    T cm = cb, sm = sb;
#pragma unroll
    for (int m = 1; m <= l; ++m) {
        const T s = sgn > 0 ? sm : -sm;
        const T x = a[l + m], y = a[l - m];
        a[l + m] = cm * x - s * y;
        a[l - m] = s * x + cm * y;
        const T cn = cm * cb - sm * sb, sn = sm * cb + cm * sb;
        cm = cn;
        sm = sn;
    }
}

// Block l of D^T (in = 1: Xm Dz(-beta) Xp Dz(-alpha)) or of D (in = 0:
// Dz(alpha) Xm Dz(beta) Xp).  Both directions share one copy of the Xp and
// Xm codelets (half the code of separate forward / backward bodies, which
// keeps the instruction working set of the solve small).
template <int l, typename T>
__device__ __forceinline__ void rot_block(T* v, int vs, const T* csa, T cb, T sb, int in) {
    constexpr int n = 2 * l + 1;
    T a[n], b[n];
#pragma unroll
    for (int j = 0; j < n; ++j) a[j] = v[(l * l + j) * vs];
    if (in) dz_block<l, T>(a, csa, -1);
    XRot<l>::template p<RotReal<T>>(a, b);
    dz_block_rec<l, T>(b, cb, sb, in ? -1 : +1);
    XRot<l>::template m<RotReal<T>>(b, a);
    if (!in) dz_block<l, T>(a, csa, +1);
#pragma unroll
    for (int j = 0; j < n; ++j) v[(l * l + j) * vs] = a[j];
}

// D^T (in = 1) or D (in = 0) on the degree blocks l set in lmask;
// cos/sin(m beta) by recurrence from (cb, sb).  Compiled once per precision.
template <typename T>
__device__ __noinline__ void rot_all(T* __restrict__ v, int vs, int L, const T* __restrict__ csa, T cb, T sb, int in,
                                     unsigned lmask) {
#pragma unroll 1
    for (int l = 0; l <= L; ++l) {
        if (!((lmask >> l) & 1u)) continue;
        switch (l) {
#define WLC_ROT(q)                              \
    case q:                                     \
        rot_block<q, T>(v, vs, csa, cb, sb, in); \
        break;
            WLC_ROT(0) WLC_ROT(1) WLC_ROT(2) WLC_ROT(3) WLC_ROT(4) WLC_ROT(5) WLC_ROT(6)
            WLC_ROT(7) WLC_ROT(8) WLC_ROT(9) WLC_ROT(10) WLC_ROT(11) WLC_ROT(12)
#undef WLC_ROT
            default:
                break;
        }
    }
}

// The rotations of the FP64 form on 64-bit integers (see wlc_fixfft.cuh for
// why and for the number format): one exponent per (kz, part, degree block),
// leading bit of the largest element at kRotTop.  A row of X has at most 7
// entries of absolute sum 2.56, so with factors of 62 fraction bits the middle
// sums stay below 2.56 * 2^61 + 7 * 2^58.3 < 2^63.
// Instruction fetch bounds straight-line code here (every instruction of a
// codelet serves one column once per direction): with conversions, rotations
// about z and X all unrolled the rotations of L = 10 were 200 kB of code and
// waited 5 cycles of 8 for instructions.  So all of it is loops: over the
// (m, -m) pairs for conversions and rotations about z, and for X over its
// four dense blocks per degree, whose factors come from a constant table; the
// block stays in the shared column in between.  One CTA's two rotations at
// L = 10, N = 64 (512 threads): 172 k clocks unrolled, 100 k as loops; FP64
// pass B with everything in this file and wlc_fixfft.cuh 3.7 -> 2.0 ms (real-8
// literals: 1.4 ms).
constexpr int kRotTop = 55;
struct FixAcc {
    long long hi, mid;
    __device__ __forceinline__ FixAcc() : hi(0), mid(kHalf) {}
    __device__ __forceinline__ void mad(fxh k, fxh v) {
        hi += (long long)v.h * k.h;
        mid += (long long)v.h * k.l;
        mid += (long long)v.l * k.h;
    }
    __device__ __forceinline__ long long done() const { return fx_join(hi, mid); }
};

// one dense block of X (t: its factors, row by row) on every second element
template <int S> __device__ __forceinline__ void x_dense(long long* v, int st, const int2* t) {
    fxh a[S];
#pragma unroll
    for (int c = 0; c < S; ++c) a[c] = halves(v[c * st]);
#pragma unroll
    for (int r = 0; r < S; ++r) {
        FixAcc s;
#pragma unroll
        for (int c = 0; c < S; ++c) s.mad(fxh{t[r * S + c].x, t[r * S + c].y}, a[c]);
        v[r * st] = s.done();
    }
}
// X (tr = 0) or its transpose (tr = 1) on block l, outputs in the inputs' places
__device__ __noinline__ void x_fx(long long* v, int vs, int l, int tr) {
#pragma unroll 1
    for (int b = 0; b < 4; ++b) {
        const int2* t = kXtab + kXdesc[l][b][2] + (tr ? kXentries : 0);
        long long* p = v + kXdesc[l][b][1] * vs;
        switch (kXdesc[l][b][0]) {
            case 1: x_dense<1>(p, 2 * vs, t); break;
            case 2: x_dense<2>(p, 2 * vs, t); break;
            case 3: x_dense<3>(p, 2 * vs, t); break;
            case 4: x_dense<4>(p, 2 * vs, t); break;
            case 5: x_dense<5>(p, 2 * vs, t); break;
            case 6: x_dense<6>(p, 2 * vs, t); break;
            case 7: x_dense<7>(p, 2 * vs, t); break;
            default: break;
        }
    }
}

// the pair (x, y) rotated by an angle with cos, sin f (sgn < 0: by minus it).
// The sign goes to the 64-bit numbers, never to the halves of the factor: a low
// half of -2^31 has no negative in 32 bits (about one random box in a thousand
// has such a sine, which then was off by 2^-30).
__device__ __forceinline__ void dz_pair_fx(long long& x, long long& y, const fxw& f, int sgn) {
    const fxh a = halves(x), b = halves(y);
    const fxh sa = sgn > 0 ? a : halves(-x), sb = sgn > 0 ? halves(-y) : b;
    FixAcc u, w;
    u.mad(f.x, a);
    u.mad(f.y, sb);
    w.mad(f.y, sa);
    w.mad(f.x, b);
    x = u.done();
    y = w.done();
}

// D^T (in = 1) or D (in = 0) on the degree blocks l set in lmask of the
// thread's word v (doubles, element i at v[i*vs]); csa[m], csb[m*ms]: cos,
// sin of m alpha and m beta
__device__ __noinline__ void rot_all_fx(double* __restrict__ v0, int vs, int L, const fxw* __restrict__ csa,
                                        const fxw* __restrict__ csb, int ms, int in, unsigned lmask) {
#pragma unroll 1
    for (int l = 1; l <= L; ++l) {  // degree 0 does not rotate
        if (!((lmask >> l) & 1u)) continue;
        double* const vd = v0 + l * l * vs;          // first element (m = -l)
        long long* const v = reinterpret_cast<long long*>(vd);
        const int mid = l * vs;                      // m = 0
        int E = 0, lift = 0;
#pragma unroll 4
        for (int j = 0; j < 2 * l + 1; ++j) E = max(E, (reinterpret_cast<const int*>(vd + j * vs)[1] >> 20) & 0x7ff);
        if (E < kExpLow) {
            E = lift_tiny(vd, vs, 2 * l + 1);
            if (E == 0) continue;  // zeros stay zeros
            lift = kLift;
        }
        if (E == 2047) E = kExpBad;
        v[mid] = d2fx<kRotTop>(vd[mid], E).v;
#pragma unroll 2
        for (int m = 1; m <= l; ++m) {
            long long x = d2fx<kRotTop>(vd[mid + m * vs], E).v, y = d2fx<kRotTop>(vd[mid - m * vs], E).v;
            if (in) dz_pair_fx(x, y, csa[m], -1);
            v[mid + m * vs] = x;
            v[mid - m * vs] = y;
        }
        x_fx(v, vs, l, 0);
#pragma unroll 2
        for (int m = 1; m <= l; ++m) {
            const int px = mid + (m + kXshift[l][m & 1][0]) * vs, py = mid + (kXshift[l][m & 1][1] - m) * vs;
            long long x = v[px], y = v[py];
            dz_pair_fx(x, y, csb[m * ms], in ? -1 : +1);
            v[px] = x;
            v[py] = y;
        }
        x_fx(v, vs, l, 1);
        E += kTop - kRotTop - lift;
        const bool rare = fx_rare(E);
        vd[mid] = rare ? fx2d_rare(v[mid], E) : fx2d_cvt(v[mid], E);
#pragma unroll 2
        for (int m = 1; m <= l; ++m) {
            long long x = v[mid + m * vs], y = v[mid - m * vs];
            if (!in) dz_pair_fx(x, y, csa[m], +1);
            vd[mid + m * vs] = rare ? fx2d_rare(x, E) : fx2d_cvt(x, E);
            vd[mid - m * vs] = rare ? fx2d_rare(y, E) : fx2d_cvt(y, E);
        }
    }
}

// Tridiagonal systems of one m (both +m and -m share the real pivots):
// d_0 = A_m, d_j = A_l + e^2/d_{j-1}, e = t z_{l-1}; forward
// y_l = b_l - i (e/d_{j-1}) y_{l-1}; back x_l = (y_l - i t z_l x_{l+1})/d_l.
template <typename T>
__device__ __noinline__ void tridiag_all(typename cvec<T>::t* __restrict__ v, int vs, int L, T t, T c0, T dcoef,
                                         const T* __restrict__ zoff, const T* __restrict__ pivrow, unsigned mmask) {
    using C = typename cvec<T>::t;
#pragma unroll 1
    for (int m = 0; m <= L; ++m) {
        if (!((mmask >> m) & 1u)) continue;
        const int n = L - m + 1;
        T dinv[16];
        // with a pivot table the inverse pivots are read from its row (L1-resident)
        // rather than copied into a runtime-indexed local array
        const T* pr = pivrow ? pivrow + m * (L + 1) - (m * (m - 1)) / 2 : dinv;
        if (!pivrow) {
            T d = c0 + dcoef * (T)(m * (m + 1));
            dinv[0] = (T)1 / d;
            for (int j = 1; j < n; ++j) {
                const int l = m + j;
                const T e = t * zoff[(l - 1) * (l - 1) + (l - 1) + m];
                d = (c0 + dcoef * (T)(l * (l + 1))) + e * (e * dinv[j - 1]);
                dinv[j] = (T)1 / d;
            }
        }
        if (m == 0) {
            int idx = 0;
            C yp = v[0];
            for (int j = 1; j < n; ++j) {
                const int prev = idx;
                idx = j * j + j;
                const T g = t * zoff[prev] * pr[j - 1];
                C y = v[idx * vs];
                y = cmk<C>(fma(g, yp.y, y.x), fma(-g, yp.x, y.y));
                v[idx * vs] = y;
                yp = y;
            }
            C xn = cmk<C>(yp.x * pr[n - 1], yp.y * pr[n - 1]);
            v[idx * vs] = xn;
            for (int j = n - 2; j >= 0; --j) {
                idx = j * j + j;
                const T e = t * zoff[idx];
                const C y = v[idx * vs];
                xn = cmk<C>(fma(e, xn.y, y.x) * pr[j], fma(-e, xn.x, y.y) * pr[j]);
                v[idx * vs] = xn;
            }
            continue;
        }
        // the +m and -m systems share couplings and pivots: both chains advance
        // in lockstep (two independent dependency chains per step)
        int ip = m * m + 2 * m, im = m * m;
        C yp = v[ip * vs], ym = v[im * vs];
        for (int j = 1; j < n; ++j) {
            const int l = m + j;
            const T g = t * zoff[ip] * pr[j - 1];
            ip = l * l + l + m;
            im = l * l + l - m;
            C y1 = v[ip * vs], y2 = v[im * vs];
            y1 = cmk<C>(fma(g, yp.y, y1.x), fma(-g, yp.x, y1.y));
            y2 = cmk<C>(fma(g, ym.y, y2.x), fma(-g, ym.x, y2.y));
            v[ip * vs] = y1;
            v[im * vs] = y2;
            yp = y1;
            ym = y2;
        }
        C xp = cmk<C>(yp.x * pr[n - 1], yp.y * pr[n - 1]);
        C xm = cmk<C>(ym.x * pr[n - 1], ym.y * pr[n - 1]);
        v[ip * vs] = xp;
        v[im * vs] = xm;
        for (int j = n - 2; j >= 0; --j) {
            const int l = m + j;
            ip = l * l + l + m;
            im = l * l + l - m;
            const T e = t * zoff[ip], p = pr[j];
            const C y1 = v[ip * vs], y2 = v[im * vs];
            xp = cmk<C>(fma(e, xp.y, y1.x) * p, fma(-e, xp.x, y1.y) * p);
            xm = cmk<C>(fma(e, xm.y, y2.x) * p, fma(-e, xm.x, y2.y) * p);
            v[ip * vs] = xp;
            v[im * vs] = xm;
        }
    }
}

// asynchronous global -> shared copy of one complex element (cp.async:
// the column loads are all in flight before the tables are staged)
template <typename C> __device__ __forceinline__ void cp_async_elem(C* sdst, const C* gsrc) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
    if constexpr (sizeof(C) == 16)
        asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
    else
        asm volatile("cp.async.ca.shared.global [%0], [%1], 8;\n" ::"r"(sa), "l"(gsrc) : "memory");
}

template <typename X> __device__ __forceinline__ void stage(X* dst, const X* src, int n) {
    for (int e = threadIdx.x; e < n; e += blockDim.x) dst[e] = src[e];
}

// registers a thread: three 256-thread CTAs of the FP32 form on an SM (their
// columns take a third of its shared memory at 64^3, L = 10), one 512-thread
// CTA of the FP64 form
template <typename T, int N, bool B = false>
__global__ void __maxnreg__(sizeof(T) == 4 ? 80 : 128)
    zfft_solve(SolveArgs<T> a0, const SolveArgs<T>* __restrict__ batch, SolveSplit split) {
    const SolveArgs<T> a = pick_args<B>(a0, batch);
    using C = typename cvec<T>::t;
    constexpr int NP = N + 1;
    const SolveTablesT<T>& g = a.tab;
    const int M = g.M, L = g.L;
    // the FP32 first-order correction exists in the FP64 path only
    const int correct = sizeof(T) == 8 ? a.correct : 0;
    const SolveSmem sm = solve_smem(N, M, L, g.ndr, sizeof(T), correct);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    C* col = reinterpret_cast<C*>(smem_raw + sm.col);
    C* tw = reinterpret_cast<C*>(smem_raw + sm.tw);
    fxw* twx = reinterpret_cast<fxw*>(smem_raw + sm.tw);
    int16_t* es = reinterpret_cast<int16_t*>(smem_raw + sm.es);
    T* csa = reinterpret_cast<T*>(smem_raw + sm.csa);
    float* csaf = reinterpret_cast<float*>(smem_raw + sm.csaf);
    T* s_zoff = reinterpret_cast<T*>(smem_raw + sm.zoff);
    float* s_zofff = reinterpret_cast<float*>(smem_raw + sm.zofff);
    int* s_drp = reinterpret_cast<int*>(smem_raw + sm.dr_ptr);
    int16_t* s_drc = reinterpret_cast<int16_t*>(smem_raw + sm.dr_col);
    float* s_drv = reinterpret_cast<float*>(smem_raw + sm.dr_valf);
    float2* corr = reinterpret_cast<float2*>(smem_raw + sm.corr);
    const int colid = blockIdx.x;
    C* gcol = a.phat + (size_t)colid * M * N;
    dep_wait<chained_step(N, sizeof(T), B)>();
    for (int e = threadIdx.x; e < M * N; e += blockDim.x) cp_async_elem(col + (e / N) * NP + (e % N), gcol + e);
    asm volatile("cp.async.commit_group;\n" ::: "memory");
    stage(s_zoff, g.zoff, M);
    if (correct) {
        stage(s_zofff, g.zofff, M);
        stage(s_drp, g.dr_ptr, M + 1);
    }
    const int kyi = colid / a.nkx, kxi = colid % a.nkx;
    const int ix = fold_n(kxi, N), iy = fold_n(kyi, N);
    const double kx = ix * a.kf[0], ky = iy * a.kf[1];
    if (correct)  // entries of dR times the column's kx, ky; bit 8 marks those still to be multiplied by kz
        for (int e = threadIdx.x; e < g.ndr; e += blockDim.x) {
            const int ax = g.dr_axis[e];
            s_drc[e] = (int16_t)(g.dr_col[e] | (ax == 2 ? 0x100 : 0));
            s_drv[e] = g.dr_valf[e] * (ax == 0 ? (float)kx : ax == 1 ? (float)ky : 1.f);
        }
    if constexpr (sizeof(T) == 8) {
        for (int e = threadIdx.x; e < N; e += blockDim.x) twx[e] = make_fxw(a.twg[e]);
    } else {
        for (int e = threadIdx.x; e < N; e += blockDim.x) tw[e] = a.twg[e];
    }
    // FP64 form: cos, sin(m beta) of every kz position as fixed-point factors
    // [m][p], and sigma ds |k| in place of m = 0
    fxw* const csb = sm.beta ? reinterpret_cast<fxw*>(smem_raw + sm.beta) : nullptr;
    if (threadIdx.x == blockDim.x - 1) {
        const double rho = sqrt(kx * kx + ky * ky);
        const double ca = rho > 0 ? kx / rho : 1.0, sa = rho > 0 ? ky / rho : 0.0;
        double cm = 1.0, sm2 = 0.0;
        for (int m = 0; m <= L; ++m) {
            if (csb) {
                reinterpret_cast<fxw*>(csa)[m] = make_fxw(make_double2(cm, sm2));
            } else {
                csa[2 * m] = (T)cm;
                csa[2 * m + 1] = (T)sm2;
            }
            csaf[2 * m] = (float)cm;
            csaf[2 * m + 1] = (float)sm2;
            const double cn = cm * ca - sm2 * sa, sn = sm2 * ca + cm * sa;
            cm = cn;
            sm2 = sn;
        }
    }
    if (csb && threadIdx.x < N) {
        const double kz = fold_n(perm_index<N>(threadIdx.x), N) * a.kf[2];
        const double rho2 = kx * kx + ky * ky, kn2 = rho2 + kz * kz;
        const double kn = sqrt(kn2), rho = sqrt(rho2);
        const double cb = kn2 > 0 ? kz / kn : 1.0, sb = kn2 > 0 ? rho / kn : 0.0;
        *reinterpret_cast<double*>(csb + threadIdx.x) = a.sigma * a.ds * kn;
        fxw f = make_fxw(make_double2(cb, sb));
        const fxw f1 = f;
        fxc z{mkfx(join_halves(f.x)), mkfx(join_halves(f.y))};
        for (int m = 1; m <= L; ++m) {
            csb[m * N + threadIdx.x] = f;
            z = fx_twiddle<-1>(z, f1);  // times e^{i beta}
            f = fxw{halves(z.x.v), halves(z.y.v)};
        }
    }
    asm volatile("cp.async.wait_group 0;\n" ::: "memory");
    __syncthreads();
    if constexpr (sizeof(T) == 8)
        fx_nat2perm<N, -1, true>(col, M, 1, NP, twx, es, es, FromDoubles{});
    else
        fft_nat2perm<N, -1>(col, M, 1, NP, tw);

    // Work split.  Rotations: thread t owns word w = t % 2N of the column
    // (kz position w / 2, real or imaginary part w % 2) and the degree blocks
    // of part t / 2N.  Tridiagonal systems (complex): kz position p = t % N
    // and the m systems of part t / N.  The parts meet at CTA barriers.
    // The parts are dealt warp by warp where a column is whole warps: with 4
    // parts the warps of one part then share a scheduler and its instruction
    // fetch (the codelets are straight-line code, each instruction used once).
    const int parts = blockDim.x / (2 * N);
    int w, lpart;
    if constexpr ((2 * N) % 32 == 0) {
        const int warp = threadIdx.x / 32;
        lpart = warp % parts;
        w = (warp / parts) * 32 + threadIdx.x % 32;
    } else {
        lpart = threadIdx.x / (2 * N);
        w = threadIdx.x % (2 * N);
    }
    const int p = threadIdx.x % N;
    const unsigned lmask = split.l[lpart], mmask = split.m[threadIdx.x / N];
    const T c0 = (T)a.c0, dcoef = (T)a.dcoef;
    const int iz = fold_n(perm_index<N, T>(p), N), izr = fold_n(perm_index<N, T>(w / 2), N);
    const double kz = iz * a.kf[2];
    // angle of k to z and sigma ds |k|: in FP64 for FP64 propagators, in FP32
    // for FP32 ones (every thread runs this, and the FP64 pipe is a small
    // fraction of the FP32 pipe)
    const int key = ix * ix + iy * iy + iz * iz;
    const T* pivrow = a.pivtab ? a.pivtab + (size_t)key * a.npiv : nullptr;
    T cb = 1, sb = 0, t;  // cos beta, sin beta of the rotations' wavevector, sigma ds |k| of the systems'
    if constexpr (sizeof(T) == 8) {
        if (csb) {
            t = *reinterpret_cast<const double*>(csb + p);
        } else {
            const double kzr = izr * a.kf[2], rho2 = kx * kx + ky * ky;
            const double rho = sqrt(rho2), kn = sqrt(rho2 + kzr * kzr);
            cb = kn > 0 ? kzr / kn : 1.0;
            sb = kn > 0 ? rho / kn : 0.0;
            t = a.sigma * a.ds * sqrt(rho2 + kz * kz);
        }
    } else {
        // every operation rounded explicitly (no contraction choices, so all
        // instantiations agree bit for bit); with a pivot table ds |k| is
        // formed from the key exactly as the table forms it
        const float kxf = __fmul_rn((float)ix, (float)a.kf[0]), kyf = __fmul_rn((float)iy, (float)a.kf[1]);
        const float kzf = __fmul_rn((float)iz, (float)a.kf[2]), kzrf = __fmul_rn((float)izr, (float)a.kf[2]);
        const float rho = __fsqrt_rn(__fadd_rn(__fmul_rn(kxf, kxf), __fmul_rn(kyf, kyf)));
        const float rho2 = __fmul_rn(rho, rho);
        const float kr = __fsqrt_rn(__fadd_rn(rho2, __fmul_rn(kzrf, kzrf)));
        const float kn = __fsqrt_rn(__fadd_rn(rho2, __fmul_rn(kzf, kzf)));
        cb = kr > 0.f ? __fdiv_rn(kzrf, kr) : 1.f;
        sb = kr > 0.f ? __fdiv_rn(rho, kr) : 0.f;
        const float tk = pivrow ? __fmul_rn((float)(a.ds * a.kf[0]), __fsqrt_rn((float)key)) : __fmul_rn((float)a.ds, kn);
        t = a.sigma > 0 ? tk : -tk;
    }
    T* vr = reinterpret_cast<T*>(col) + w;
    auto rotate = [&](int in) {
        if constexpr (sizeof(T) == 8) {
            if (csb) return rot_all_fx(vr, 2 * NP, L, reinterpret_cast<const fxw*>(csa), csb + w / 2, N, in, lmask);
        }
        rot_all<T>(vr, 2 * NP, L, csa, cb, sb, in, lmask);
    };
    float cbf, sbf;  // of the correction (csb may lie in its space)
    if constexpr (sizeof(T) == 8) {
        if (csb) {
            const fxw f = csb[(L > 0 ? N : 0) + w / 2];
            cbf = (float)((double)join_halves(f.x) * 0x1p-62);
            sbf = (float)((double)join_halves(f.y) * 0x1p-62);
        } else {
            cbf = (float)cb;
            sbf = (float)sb;
        }
    }
    rotate(1);
    __syncthreads();
    tridiag_all<T>(col + p, NP, L, t, c0, dcoef, s_zoff, pivrow, mmask);
    __syncthreads();
    rotate(0);
    __syncthreads();
    if (correct) {
        // x -= G_cov^-1 (i sigma ds (k . dR) x), in FP32; times i: the real
        // part takes the sums over the imaginary parts and the other way
        // round.  x goes through the correction's space as floats, the sums
        // wait in local memory until every thread has read it.
        const float sds = (w & 1) ? (float)(a.sigma * a.ds) : -(float)(a.sigma * a.ds);
        const float kzr = (float)(izr * a.kf[2]);
        float* const r = reinterpret_cast<float*>(corr) + w;
        const float* const xo = reinterpret_cast<const float*>(corr) + (w ^ 1);
        for (int l = 0; l <= L; ++l) {
            if (!((lmask >> l) & 1u)) continue;
#pragma unroll 4
            for (int i = l * l; i < (l + 1) * (l + 1); ++i) r[i * 2 * N] = d2f((double)vr[i * 2 * NP]);
        }
        __syncthreads();
        float sums[(kRotLmax + 1) * (kRotLmax + 1)];
        int ns = 0;
        for (int l = 0; l <= L; ++l) {
            if (!((lmask >> l) & 1u)) continue;
            for (int i = l * l; i < (l + 1) * (l + 1); ++i) {
                float sum = 0.f;
                const int e1 = s_drp[i + 1];
#pragma unroll 4
                for (int e = s_drp[i]; e < e1; ++e) {
                    const int c = s_drc[e];
                    const float g = c & 0x100 ? s_drv[e] * kzr : s_drv[e];
                    sum = fmaf(g, xo[(c & 0xff) * 2 * N], sum);
                }
                sums[ns++] = sds * sum;
            }
        }
        __syncthreads();
        ns = 0;
        for (int l = 0; l <= L; ++l) {
            if (!((lmask >> l) & 1u)) continue;
            for (int i = l * l; i < (l + 1) * (l + 1); ++i) r[i * 2 * N] = sums[ns++];
        }
        rot_all<float>(r, 2 * N, L, csaf, cbf, sbf, 1, lmask);
        __syncthreads();
        tridiag_all<float>(corr + p, N, L, (float)t, (float)a.c0, (float)a.dcoef, s_zofff, nullptr, mmask);
        __syncthreads();
        rot_all<float>(r, 2 * N, L, csaf, cbf, sbf, 0, lmask);
    }
    __syncthreads();
    if constexpr (sizeof(T) == 8) {
        if (correct)
            fx_perm2nat<N, +1, true>(col, M, 1, NP, twx, es, es, FromDoublesLess{corr, N});
        else
            fx_perm2nat<N, +1, true>(col, M, 1, NP, twx, es, es, FromDoubles{});
    } else
        fft_perm2nat<N, +1>(col, M, 1, NP, tw);
    dep_next<chained_step(N, sizeof(T), B)>();
    if (a.split) {
        // Crank-Nicolson operator (I + ds/2 A)^-1 (I - ds/2 A) = 2 (I + ds/2 A)^-1 - I
        // applied through the z transforms: IFFT_z(2x - b) = 2 IFFT_z(x) - N b,
        // with b the column as pass A wrote it (still in phat)
        for (int e = threadIdx.x; e < M * N; e += blockDim.x) {
            const C x = col[(e / N) * NP + (e % N)], b = gcol[e];
            gcol[e] = cmk<C>(fma((T)2, x.x, -(T)N * b.x), fma((T)2, x.y, -(T)N * b.y));
        }
    } else {
        for (int e = threadIdx.x; e < M * N; e += blockDim.x) gcol[e] = col[(e / N) * NP + (e % N)];
    }
}

// inverse pivots 1/d_j of the tridiagonal systems for every key
// ix^2+iy^2+iz^2 <= nkeys-1 (isotropic spacing), one (order, block)
template <typename T>
__global__ void pivot_table(T* out, int nkeys, int L, double c0, double dcoef, double ds, double kf,
                            const T* __restrict__ zoff) {
    const int npiv = (L + 1) * (L + 2) / 2;
    for (int key = blockIdx.x * blockDim.x + threadIdx.x; key < nkeys; key += gridDim.x * blockDim.x) {
        // ds |k| as the solve kernel forms it for this precision
        T t;
        if constexpr (sizeof(T) == 8)
            t = ds * kf * sqrt((double)key);
        else
            t = __fmul_rn((float)(ds * kf), __fsqrt_rn((float)key));
        T* row = out + (size_t)key * npiv;
        for (int m = 0; m <= L; ++m) {
            T* pr = row + m * (L + 1) - (m * (m - 1)) / 2;
            T d = (T)c0 + (T)dcoef * (T)(m * (m + 1));
            T dinv = (T)1 / d;
            pr[0] = dinv;
            for (int j = 1; j <= L - m; ++j) {
                const int l = m + j;
                const T e = t * zoff[(l - 1) * (l - 1) + (l - 1) + m];
                d = ((T)c0 + (T)dcoef * (T)(l * (l + 1))) + e * (e * dinv);
                dinv = (T)1 / d;
                pr[j] = dinv;
            }
        }
    }
}

template <typename T> size_t solve_smem_bytes(const SolveArgs<T>& a) {
    const int N = 2 * (a.nkx - 1);
    return solve_smem(N, a.tab.M, a.tab.L, a.tab.ndr, sizeof(T), a.correct).total;
}

// Work split of the solve: greedy balance of the degree blocks over P parts
// and of the m systems over 2P.  threads = N P as the tuner counts them (0:
// by the rule below); the CTA has 2 N P threads.
//
// Rule: as many parts as still leave few waves.  A CTA's time is about 0.65
// (loads, FFTs) + the largest part's share of the solve; the columns of the
// launch come in waves of the CTAs that fit the SMs (shared memory; 80
// registers a thread in FP32, 128 in FP64).  The estimate names the measured
// best split, or one within 8 % of it, for N = 16..128 in both precisions;
// one fixed thread count cost up to 2.2x (FP64 24^3, L = 5: 4 waves, 150 us;
// 3 parts, one wave: 67 us).
template <typename T> static int solve_parts(int N, int L, int threads, size_t smem, int columns) {
    const int pmax = kSolveThreads / N < 1 ? 1 : kSolveThreads / N;
    if (threads > 0) return std::min(std::max(threads / N, 1), pmax);
    const int fit_smem = std::max(1, (int)(227 * 1024 / (smem + 1024)));
    const float total = (L + 1) * (L * (2 * L + 1) / 6.0f + 1.5f * L + 1.0f), top = (float)(L * L + 3 * L + 1);
    int best = 1;
    float tbest = 1e30f;
    for (int p = 1; p <= std::min(pmax, L + 1); ++p) {
        const int warps = (2 * N * p + 31) / 32;
        const int fit = std::max(1, std::min(fit_smem, (sizeof(T) == 4 ? 25 : 16) / warps));
        const int waves = (columns + 152 * fit - 1) / (152 * fit);
        const float t = (float)waves * (0.65f + std::max(1.0f / p, top / total) + 0.01f * p);
        if (t < tbest) {
            tbest = t;
            best = p;
        }
    }
    return best;
}
static SolveSplit solve_split(int L, int parts) {
    SolveSplit s{};
    auto deal = [](uint16_t* mask, int n, int first, int step, int count, auto cost) {
        float load[2 * kSolveParts] = {};
        for (int k = 0, x = first; k < count; ++k, x += step) {
            int best = 0;
            for (int q = 1; q < n; ++q)
                if (load[q] < load[best]) best = q;
            mask[best] |= (uint16_t)(1u << x);
            load[best] += cost(x);
        }
    };
    deal(s.l, parts, L, -1, L + 1, [](int l) { return (float)(l * l + 3 * l + 1); });  // costliest first
    deal(s.m, 2 * parts, 0, 1, L + 1, [L](int m) { return (float)((L - m + 1) * (m > 0 ? 2 : 1)); });
    return s;
}

template <typename T, int N> static cudaError_t launch_solve_n(const SolveArgs<T>& a, cudaStream_t st, int threads) {
    if (const cudaError_t e = smem_attr_once((const void*)zfft_solve<T, N>, 227 * 1024); e != cudaSuccess) return e;
    const size_t smem = solve_smem_bytes<T>(a);
    const int parts = solve_parts<T>(N, a.tab.L, threads, smem, a.nkx * N);
    return launch_chained(chained_step(N, sizeof(T), false), zfft_solve<T, N>, dim3(a.nkx * N), 2 * N * parts, smem, st, a, nullptr,
                          solve_split(a.tab.L, parts));
}

template <typename T> cudaError_t launch_solve(int N, const SolveArgs<T>& a, cudaStream_t st, int threads) {
    switch (N) {
#define WLC_CASE(n) \
    case n:         \
        return launch_solve_n<T, n>(a, st, threads);
        WLC_FOR_EACH_N(WLC_CASE)
#undef WLC_CASE
        default:
            return cudaErrorInvalidValue;
    }
}

template <int N> static cudaError_t set_solve_batched_attr() {
    return smem_attr_once((const void*)zfft_solve<float, N, true>, 227 * 1024);
}

template <int N> static cudaError_t launch_solve_batched_n(const BatchLaunch<float>& b, cudaStream_t st) {
    if (const cudaError_t e = set_solve_batched_attr<N>(); e != cudaSuccess) return e;
    const int parts = solve_parts<float>(N, b.lmax, b.solve_threads, b.solve_smem, b.nkx * N * b.count);
    return launch_chained(chained_step(N, 4, true), zfft_solve<float, N, true>, dim3(b.nkx * N, 1, b.count), 2 * N * parts, b.solve_smem, st,
                          SolveArgs<float>{}, b.dsolve, solve_split(b.lmax, parts));
}

cudaError_t launch_solve_batched(int N, const BatchLaunch<float>& b, cudaStream_t st) {
    switch (N) {
#define WLC_CASE(n) \
    case n:         \
        return launch_solve_batched_n<n>(b, st);
        WLC_FOR_EACH_BATCH_N(WLC_CASE)
#undef WLC_CASE
        default:
            return cudaErrorInvalidValue;
    }
}

cudaError_t prepare_solve_batched(int N) {
    switch (N) {
#define WLC_CASE(n) \
    case n:         \
        return set_solve_batched_attr<n>();
        WLC_FOR_EACH_BATCH_N(WLC_CASE)
#undef WLC_CASE
        default:
            return cudaErrorInvalidValue;
    }
}

template <typename T>
cudaError_t launch_pivot_table(T* out, int nkeys, int L, double c0, double dcoef, double ds, double kf, const T* zoff,
                               cudaStream_t st) {
    pivot_table<T><<<(nkeys + 127) / 128, 128, 0, st>>>(out, nkeys, L, c0, dcoef, ds, kf, zoff);
    return cudaGetLastError();
}

template cudaError_t launch_solve<double>(int, const SolveArgs<double>&, cudaStream_t, int);
template cudaError_t launch_solve<float>(int, const SolveArgs<float>&, cudaStream_t, int);
template size_t solve_smem_bytes<double>(const SolveArgs<double>&);
template size_t solve_smem_bytes<float>(const SolveArgs<float>&);
template cudaError_t launch_pivot_table<double>(double*, int, int, double, double, double, double, const double*,
                                                cudaStream_t);
template cudaError_t launch_pivot_table<float>(float*, int, int, double, double, double, double, const float*,
                                               cudaStream_t);

}  // namespace wlc
