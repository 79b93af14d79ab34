// wlc_step.cu -- kernels of one contour step (passes A, B, C; see
// wlc_kernels.cuh) and their host launchers, instantiated for every
// supported grid edge N and for FP64 / FP32.
#include <cstdio>

#include "wlc_attr.h"
#include "wlc_fixfft.cuh"
#include "wlc_kernels.cuh"
#include "wlc_step.h"

namespace wlc {

__device__ __forceinline__ int fold_idx(int i, int n) { return i <= n / 2 ? i : i - n; }

// BDF right-hand side at grid point r of coefficient i (init_pr,
// MDE_ABC.f90:245-375): order 1 (1 - ds w) q1; order 2
// 2 q1 - q2/2 - ds w (2 q1 - q2); order 3 sum_j c_j(r) q_j with
// c = (3 - 3 ds w, -3/2 + 3 ds w, 1/3 - ds w) precomputed per block.
// FP32 form (the same for every launch variant): dw = ds w(r) rounded once, every operation rounded explicitly.
// Split-scheme steps (kSplitOrder) pass e^{-w ds/2} as dw: q1 e^{-w ds/2}.
__device__ __forceinline__ float rhs_f32(int order, float q1, float q2, float q3, float dw, float third) {
    if (order == 0) return q1;
    if (order == kSplitOrder) return __fmul_rn(dw, q1);
    if (order == 1) return __fmul_rn(__fsub_rn(1.0f, dw), q1);
    if (order == 2) {
        const float t = __fsub_rn(__fmul_rn(2.0f, q1), q2);
        return __fsub_rn(__fsub_rn(__fmul_rn(2.0f, q1), __fmul_rn(0.5f, q2)), __fmul_rn(dw, t));
    }
    const float dw3 = __fmul_rn(3.0f, dw);
    const float c1 = __fsub_rn(3.0f, dw3), c2 = __fadd_rn(-1.5f, dw3), c3 = __fsub_rn(third, dw);
    return __fmaf_rn(c3, q3, __fmaf_rn(c2, q2, __fmul_rn(c1, q1)));
}

template <typename T, int NR>
__device__ __forceinline__ T rhs_value(const StepArgs<T>& a, size_t off, size_t r) {
    if constexpr (sizeof(T) == 4) {
        const int o = a.order;
        const int nh = hist_slices(o);
        float v = rhs_f32(o, a.h1[off], nh >= 2 ? a.h2[off] : 0.0f, nh >= 3 ? a.h3[off] : 0.0f,
                          o >= 1 ? a.dsw[r] : 0.0f, a.third);
        if (a.msterm) v += a.msterm[off];
        return v;
    }
    T v;
    if (a.order == 0) {
        v = a.h1[off];
    } else if (a.order == kSplitOrder) {  // e^{-w ds/2} q(s-1)
        v = a.cf[r] * a.h1[off];
    } else if (a.order == 1) {
        const T W = (T)a.wb[r];
        v = ((T)1 - a.ds * W) * a.h1[off];
    } else if (a.order == 2) {
        const T W = (T)a.wb[r];
        const T q1 = a.h1[off], q2 = a.h2[off];
        v = (T)2 * q1 - (T)0.5 * q2 - a.ds * W * ((T)2 * q1 - q2);
    } else {
        v = a.cf[r] * a.h1[off];
        v = fma(a.cf[NR + r], a.h2[off], v);
        v = fma(a.cf[2 * (size_t)NR + r], a.h3[off], v);
    }
    if (a.msterm) v += a.msterm[off];
    return v;
}

// rhs_value for four consecutive points (FP32; off and r multiples of 4)
__device__ __forceinline__ float4 ld4(const float* p) { return *reinterpret_cast<const float4*>(p); }
__device__ __forceinline__ float4 rhs_f32x4(const StepArgs<float>& a, size_t off, size_t r) {
    const int o = a.order;
    const int nh = hist_slices(o);
    const float4 z4 = make_float4(0.f, 0.f, 0.f, 0.f);
    const float4 q1 = ld4(a.h1 + off);
    const float4 q2 = nh >= 2 ? ld4(a.h2 + off) : z4;
    const float4 q3 = nh >= 3 ? ld4(a.h3 + off) : z4;
    const float4 dw = o >= 1 ? ld4(a.dsw + r) : z4;
    float4 v = make_float4(rhs_f32(o, q1.x, q2.x, q3.x, dw.x, a.third), rhs_f32(o, q1.y, q2.y, q3.y, dw.y, a.third),
                           rhs_f32(o, q1.z, q2.z, q3.z, dw.z, a.third), rhs_f32(o, q1.w, q2.w, q3.w, dw.w, a.third));
    if (a.msterm) {
        const float4 m = ld4(a.msterm + off);
        v.x += m.x;
        v.y += m.y;
        v.z += m.z;
        v.w += m.w;
    }
    return v;
}

// ------------------------------------------------------- async copies
__device__ __forceinline__ void cp_async16(void* sdst, const void* gsrc) {
    const unsigned sa = (unsigned)__cvta_generic_to_shared(sdst);
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(sa), "l"(gsrc) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;\n" ::: "memory"); }

// The half-spectrum planes of a CTA are kept z-fastest, out[(ky*NKX + kx)*Z + zz],
// so that the Z values of one (col, i) run in phat move as one 32-byte chunk.

// ------------------------------------------------ FP64 form: passes A and C
// x-FFTs of ZB planes of packed row pairs (zb: ZB consecutive (N/2) x N
// blocks, row stride xrow(N)), split into two half spectra each: planes zz0 ..
// zz0+ZB-1 of out (the y-FFTs of all planes follow in one batched call), as
// fixed-point numbers (twice their value) with one exponent per row pair in el
template <int N, int Z, int ZB>
__device__ __forceinline__ void fwd_x_planes_fx(double2* zb, fxc* out, int zz0, const fxw* tw, int16_t* es, int16_t* el) {
    constexpr int NKX = N / 2 + 1;
    constexpr int XR = xrow(N);
    fx_nat2perm<N, -1, false>(zb, ZB * (N / 2), 1, XR, tw, es, el + zz0 * (N / 2), FromDoubles{});
    for (int t = threadIdx.x; t < ZB * (N / 2) * NKX; t += blockDim.x) {
        const int q = t / ((N / 2) * NKX), e = t % ((N / 2) * NKX);
        const int p = e / NKX, k = e % NKX;
        const fxc* zq = reinterpret_cast<const fxc*>(zb) + (size_t)q * xplane(N);
        const fxc zk = zq[p * XR + perm_pos<N>(k)];
        const fxc zm = zq[p * XR + perm_pos<N>((N - k) % N)];
        out[((2 * p) * NKX + k) * Z + zz0 + q] = fxc{zk.x + zm.x, zk.y - zm.y};
        out[((2 * p + 1) * NKX + k) * Z + zz0 + q] = fxc{zk.y + zm.y, zm.x - zk.x};
    }
    __syncthreads();
}

// one Z-run per (ky, kx) from the half spectra to phat, in 16-byte pieces
// when a run is a whole number of them (shared reads contiguous per lane)
template <typename T, int N, int Z>
__device__ __forceinline__ void store_phat(const StepArgs<T>& a, const typename cvec<T>::t* out, int i, int z0) {
    using C = typename cvec<T>::t;
    constexpr int NKX = N / 2 + 1;
    constexpr int CH = (Z * (int)sizeof(C)) % 16 == 0 ? (Z * (int)sizeof(C)) / 16 : 0;
    for (int e = threadIdx.x; e < N * NKX; e += blockDim.x) {
        const int ky = e / NKX, kx = e % NKX;
        const size_t colid = (size_t)ky * NKX + kx;
        C* dst = a.phat + (colid * a.M + i) * N + z0;
        const C* src = out + (size_t)(perm_pos<N>(ky) * NKX + kx) * Z;
        if constexpr (CH > 0) {
#pragma unroll
            for (int q = 0; q < CH; ++q) reinterpret_cast<uint4*>(dst)[q] = reinterpret_cast<const uint4*>(src)[q];
        } else {
#pragma unroll
            for (int zz = 0; zz < Z; ++zz) dst[zz] = src[zz];
        }
    }
}

// ---------------------------------------------------------------- pass A
// V: launch variant, bit 0 half the planes per CTA, bit 1 the x-FFTs of all
// planes in one batched call (one packed-row buffer per plane)
template <typename T, int N, int V> struct XyShape {
    static constexpr int Z = xy_planes(N, sizeof(T), V & 1);
    static constexpr int ZB = (V & 2) ? Z : 1;
};

template <int N, int V = 0>
__global__ void __launch_bounds__(512) rhs_fft_xy(StepArgs<double> a) {
    using T = double;
    using C = double2;
    constexpr int Z = XyShape<T, N, V>::Z, ZB = XyShape<T, N, V>::ZB;
    constexpr int NKX = N / 2 + 1;
    constexpr int NR = N * N * N;
    constexpr int PB = (N / 2) * N;  // packed row pairs per plane
    constexpr int XR = xrow(N), PBS = xplane(N);
    extern __shared__ __align__(16) unsigned char smem_raw[];
    fxw* twx = reinterpret_cast<fxw*>(smem_raw);
    C* zb = reinterpret_cast<C*>(twx + N);  // ZB x (N/2) x N packed row pairs (row stride XR)
    C* out = zb + (size_t)ZB * PBS;         // N x NKX x Z half spectra
    int16_t* el = reinterpret_cast<int16_t*>(out + (size_t)Z * N * NKX);  // exponents per line, then scratch
    int16_t* es = el + Z * NKX;
    const int i = blockIdx.y;
    const int z0 = blockIdx.x * Z;
    for (int e = threadIdx.x; e < N; e += blockDim.x) twx[e] = make_fxw(a.twg[e]);
    dep_wait<chained_step(N, 8, false)>();
    for (int zz0 = 0; zz0 < Z; zz0 += ZB) {
        for (int t = threadIdx.x; t < ZB * PB; t += blockDim.x) {
            const int q = t / PB, e = t % PB;
            const int p = e / N, x = e % N;
            const size_t ra = ((size_t)(z0 + zz0 + q) * N + 2 * p) * N + x, rb = ra + N;
            const T va = rhs_value<T, NR>(a, (size_t)i * NR + ra, ra);
            const T vb = rhs_value<T, NR>(a, (size_t)i * NR + rb, rb);
            zb[(size_t)q * PBS + p * XR + x] = cmk<C>(va, vb);
        }
        __syncthreads();
        fwd_x_planes_fx<N, Z, ZB>(zb, reinterpret_cast<fxc*>(out), zz0, twx, es, el);
    }
    // the half spectra hold twice their value: exponent - 1
    fx_nat2perm<N, -1, true>(out, NKX * Z, NKX * Z, 1, twx, es, es, from_fixed([=](int line, int y) {
                                 return el[(line % Z) * (N / 2) + (y >> 1)] - 1;
                             }));
    dep_next<chained_step(N, 8, false)>();
    store_phat<T, N, Z>(a, out, i, z0);
}

// ---------------------------------------------------------------- pass C
__host__ __device__ constexpr int ilog2(int n) { return n > 1 ? 1 + ilog2(n / 2) : 0; }

// element k of the packed row ra + i rb, from the half spectra of its two real
// rows (element k at [k * Z]); the imaginary parts at kx = 0 and N/2 are
// discarded (c2r)
template <int N, typename K> __device__ __forceinline__ K hermitian_pair(const K* ra, const K* rb, int k, int Z) {
    K xa, xb;
    if (k <= N / 2) {
        xa = ra[k * Z];
        xb = rb[k * Z];
        if (k == 0 || k == N / 2) {
            xa.y = decltype(xa.y)(0.0);
            xb.y = decltype(xb.y)(0.0);
        }
    } else {
        xa = ra[(N - k) * Z];
        xb = rb[(N - k) * Z];
        xa.y = -xa.y;
        xb.y = -xb.y;
    }
    return cmk<K>(xa.x - xb.y, xa.y + xb.x);
}

template <int N, int V = 0> __global__ void __launch_bounds__(512) ifft_xy(StepArgs<double> a) {
    using T = double;
    using C = double2;
    constexpr int Z = XyShape<T, N, V>::Z, ZB = XyShape<T, N, V>::ZB;
    constexpr int NKX = N / 2 + 1;
    constexpr int NR = N * N * N;
    constexpr int PB = (N / 2) * N;
    constexpr int XR = xrow(N), PBS = xplane(N);
    static_assert(PBS % 2 == 0, "the half-spectrum buffer must stay 16-byte aligned");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    fxw* twx = reinterpret_cast<fxw*>(smem_raw);
    C* zb = reinterpret_cast<C*>(twx + N);  // packed row pairs, row stride XR
    C* out = zb + (size_t)ZB * PBS;
    int16_t* el = reinterpret_cast<int16_t*>(out + (size_t)Z * N * NKX);  // exponents per line, then scratch
    int16_t* es = el + Z * NKX;
    const int i = blockIdx.y;
    const int z0 = blockIdx.x * Z;
    for (int e = threadIdx.x; e < N; e += blockDim.x) twx[e] = make_fxw(a.twg[e]);
    dep_wait<chained_step(N, 8, false)>();
    // 1/N^3 is a shift of the exponents where N is a power of two
    constexpr bool kPow2 = (N & (N - 1)) == 0;
    constexpr int kShift = kPow2 ? 3 * ilog2(N) : 0;
    // all loads issued up front: one Z-run (Z * sizeof(C) bytes) per (ky, kx)
    for (int e = threadIdx.x; e < N * NKX * Z; e += blockDim.x) {
        const int col = e / Z, q = e % Z;
        cp_async16(out + (size_t)col * Z + q, a.phat + ((size_t)col * a.M + i) * N + z0 + q);
    }
    cp_async_wait_all();
    __syncthreads();
    // along y for every plane; row y now at perm_pos(y)
    fx_nat2perm<N, +1, false>(out, NKX * Z, NKX * Z, 1, twx, es, el, FromDoubles{});
    for (int zz0 = 0; zz0 < Z; zz0 += ZB) {
        // Hermitian extension of rows (2p, 2p+1) packed as one complex row;
        // the imaginary parts at kx = 0 and N/2 are discarded (c2r)
        // plane index fastest across the lanes: the ZB values read per
        // (row, k) are adjacent in out
        for (int t = threadIdx.x; t < ZB * PB; t += blockDim.x) {
            const int q = t % ZB, e = t / ZB;
            const int zz = zz0 + q;
            const int p = e / N, k = e % N;
            const fxc* ra = reinterpret_cast<const fxc*>(out) + (size_t)perm_pos<N>(2 * p) * NKX * Z + zz;
            const fxc* rb = reinterpret_cast<const fxc*>(out) + (size_t)perm_pos<N>(2 * p + 1) * NKX * Z + zz;
            reinterpret_cast<fxc*>(zb)[(size_t)q * PBS + p * XR + k] = hermitian_pair<N>(ra, rb, k, Z);
        }
        __syncthreads();
        // along x; x at perm_pos(x)
        fx_nat2perm<N, +1, true>(zb, ZB * (N / 2), 1, XR, twx, es, es, from_fixed([=](int line, int k) {
                                     return el[(k <= N / 2 ? k : N - k) * Z + zz0 + line / (N / 2)] - kShift;
                                 }));
        if (zz0 + ZB >= Z) dep_next<chained_step(N, 8, false)>();
        // packed row pair p holds rows 2p (real part) and 2p+1 (imaginary part)
        for (int t = threadIdx.x; t < ZB * PB; t += blockDim.x) {
            const int q = t / PB, e = t % PB;
            const int p = e / N, x = e % N;
            C v = zb[(size_t)q * PBS + p * XR + perm_pos<N>(x)];
            if constexpr (!kPow2) v = cscale(v, a.minv);
            const size_t r = (size_t)(z0 + zz0 + q) * N * N + (size_t)(2 * p) * N + x;
            T* dst = a.qout + (size_t)i * NR + r;
            if (a.post) {  // split scheme: the second field half step
                dst[0] = v.x * a.post[r];
                dst[N] = v.y * a.post[r + N];
            } else {
                dst[0] = v.x;
                dst[N] = v.y;
            }
        }
        __syncthreads();
    }
}

// ------------------------------------------------ FP32 form: passes A and C
// The split of a packed row pair into its two half spectra (pass A) and the
// Hermitian extension (pass C) happen in the loads of the next direction's
// first sub-pass, and the last sub-pass writes to global memory: 9 and 8
// shared-memory accesses of 8 bytes per complex point (12 with separate
// split, pack and copy-out loops), which with the barriers between them bound
// both passes.  A length N = R J is done as J transforms of length R over
// elements n J + j (twiddle w^(j k)), then R transforms of length J over j.
// Loading pass A's right-hand side straight into the first sub-pass was not
// faster (32-byte pieces cost the L1 tags four times the 16-byte vectors').
// 64^3, L = 10: pass A 171 -> 147 us, pass C 109 -> 89 us; 128^3, L = 12: 2.65 ->
// 2.42 and 1.70 -> 1.23 ms; 24^3, L = 8: 14.0 -> 11.1 and 12.2 -> 9.7 us.

// x lines: J transforms of length R over elements n J + j, then R of length J,
// the first radix first as along y and z, whichever pass it is (the order of
// the additions, and with it every bit of an FP32 result, depends on it).
// Pass A: in place, element (n, j) and output n + R j at slot n S + j.  J a
// multiple of 4: S odd, lanes j-fastest (the four elements of a 16-byte vector
// stay together).  Other J: natural order in rows of odd length, lanes
// line-fastest.  Pass C: slot (j, k) at j S + k, S odd, so that neighbouring
// lanes write >= 4 neighbours of a row.  Either way neighbouring lanes are on
// distinct banks in both sub-passes.  (Pass A with the second radix first, every
// row padded: 32^3, L = 8 18.4 us a launch against 17.5, 48^3 54.5 against 53.5,
// 96^3, L = 6 272 against 267, the others within 1 %.)
template <int N, bool FWD> struct XLine {
    static constexpr int R = Plan<N, float>::N1, J = Plan<N, float>::N2;
    static constexpr bool JFAST = J % 4 == 0;
    static constexpr int S = !FWD ? R | 1 : JFAST ? J | 1 : J;
    static constexpr int ROW = !FWD ? J * S : JFAST ? R * S : N + 1;
    __device__ __forceinline__ static int out_at(int k) { return (k % R) * S + k / R; }  // pass A, output k
};
// row length that holds either pass's lines
template <int N> __host__ __device__ constexpr int xrow32() {
    return XLine<N, true>::ROW > XLine<N, false>::ROW ? XLine<N, true>::ROW : XLine<N, false>::ROW;
}
__host__ inline int xrow32_of(int N) {
    switch (N) {
#define WLC_CASE(n) \
    case n:         \
        return xrow32<n>();
        WLC_FOR_EACH_N(WLC_CASE)
#undef WLC_CASE
        default:
            return 0;
    }
}

template <int R, int DIR> __device__ __forceinline__ void twiddles(float2* v, int j, const float2* tw) {
#pragma unroll
    for (int k = 1; k < R; ++k)
        if (j != 0) v[k] = cmul(v[k], twid<DIR>(tw, j * k));
}

// second sub-pass of the y lines in place, f(line, ky, value) for every output
template <int N, int DIR, int Z, typename F> __device__ __forceinline__ void y_second(float2* out, F&& f) {
    constexpr int NKX = N / 2 + 1, LS = NKX * Z, R = Plan<N, float>::N1, J = Plan<N, float>::N2;
    for (LineWalk it(LS); it.j < R; it.next()) {
        float2 v[J];
#pragma unroll
        for (int j = 0; j < J; ++j) v[j] = out[(j * R + it.j) * LS + it.b];
        Dft<J>::template run<DIR>(v);
#pragma unroll
        for (int k2 = 0; k2 < J; ++k2) f(it.b, it.j + R * k2, v[k2]);
    }
}

template <int N, bool B = false, int V = 0>
__global__ void __launch_bounds__(512) rhs_fft_xy32(StepArgs<float> a0, const StepArgs<float>* __restrict__ batch) {
    const StepArgs<float> a = pick_args<B>(a0, batch);
    constexpr int Z = XyShape<float, N, V>::Z, ZB = XyShape<float, N, V>::ZB;
    constexpr int NKX = N / 2 + 1, LS = NKX * Z, NR = N * N * N;
    using X = XLine<N, true>;
    constexpr int R = X::R, J = X::J;
    static_assert(X::S == J || J % 4 == 0, "four consecutive x must lie on consecutive slots");
    // item w of n x lines -> (line, n), the latter below n
    auto item = [](int w, int n) {
        if constexpr (X::JFAST) return int2{w / n, w % n};
        return int2{w % (ZB * (N / 2)), w / (ZB * (N / 2))};
    };
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* tw = reinterpret_cast<float2*>(smem_raw);
    float2* zb = tw + N;                             // [ZB][N/2] packed row pairs, X::ROW each
    float2* out = zb + (size_t)ZB * (N / 2) * X::ROW;  // [N][NKX][Z]
    const int i = blockIdx.y, z0 = blockIdx.x * Z;
    for (int e = threadIdx.x; e < N; e += blockDim.x) tw[e] = a.twg[e];
    dep_wait<chained_step(N, 4, B)>();
    __syncthreads();
    for (int zz0 = 0; zz0 < Z; zz0 += ZB) {
        // four consecutive x per thread: 16-byte loads of the history, ds*w and
        // Theta planes; the four shared stores go out in an order rotated by
        // lane, which spreads a warp over the banks
        for (int t = threadIdx.x; t < ZB * (N / 2) * (N / 4); t += blockDim.x) {
            const int b = t / (N / 4), x = 4 * (t % (N / 4));  // b = q N/2 + p
            const size_t ra = ((size_t)(z0 + zz0 + b / (N / 2)) * N + 2 * (b % (N / 2))) * N + x, rb = ra + N;
            const float4 va = rhs_f32x4(a, (size_t)i * NR + ra, ra);
            const float4 vb = rhs_f32x4(a, (size_t)i * NR + rb, rb);
            float2* zq = zb + (size_t)b * X::ROW + (x / J) * X::S + x % J;
            const int rot = (t >> 2) & 3;
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const int c = (s + rot) & 3;
                zq[c] = make_float2(c == 0 ? va.x : c == 1 ? va.y : c == 2 ? va.z : va.w,
                                    c == 0 ? vb.x : c == 1 ? vb.y : c == 2 ? vb.z : vb.w);
            }
        }
        __syncthreads();
        for (int w = threadIdx.x; w < ZB * (N / 2) * J; w += blockDim.x) {
            const int2 t = item(w, J);
            float2* row = zb + (size_t)t.x * X::ROW + t.y;
            float2 v[R];
#pragma unroll
            for (int n = 0; n < R; ++n) v[n] = row[n * X::S];
            Dft<R>::template run<-1>(v);
            twiddles<R, -1>(v, t.y, tw);
#pragma unroll
            for (int n = 0; n < R; ++n) row[n * X::S] = v[n];
        }
        __syncthreads();
        if constexpr (J > 1) {
            for (int w = threadIdx.x; w < ZB * (N / 2) * R; w += blockDim.x) {
                const int2 t = item(w, R);
                float2* row = zb + (size_t)t.x * X::ROW + t.y * X::S;
                float2 v[J];
#pragma unroll
                for (int j = 0; j < J; ++j) v[j] = row[j];
                Dft<J>::template run<-1>(v);
#pragma unroll
                for (int j = 0; j < J; ++j) row[j] = v[j];
            }
            __syncthreads();
        }
        // first y sub-pass on the half spectra of rows (2p, 2p+1): lines (kx, plane)
        for (LineWalk it(NKX * ZB); it.j < J; it.next()) {
            const int q = it.b % ZB, kx = it.b / ZB;
            const float2* zk = zb + (size_t)q * (N / 2) * X::ROW + X::out_at(kx);
            const float2* zm = zb + (size_t)q * (N / 2) * X::ROW + X::out_at((N - kx) % N);
            float2 v[R];
#pragma unroll
            for (int n = 0; n < R; ++n) {
                const int y = n * J + it.j;
                const float2 c = zk[(y >> 1) * X::ROW], d = zm[(y >> 1) * X::ROW];
                v[n] = (y & 1) ? make_float2(0.5f * (c.y + d.y), 0.5f * (d.x - c.x))
                               : make_float2(0.5f * (c.x + d.x), 0.5f * (c.y - d.y));
            }
            Dft<R>::template run<-1>(v);
            twiddles<R, -1>(v, it.j, tw);
            float2* o = out + (size_t)it.j * R * LS + kx * Z + zz0 + q;
#pragma unroll
            for (int k = 0; k < R; ++k) o[k * LS] = v[k];
        }
        __syncthreads();
    }
    dep_next<chained_step(N, 4, B)>();
    y_second<N, -1, Z>(out, [&](int b, int ky, float2 v) {
        a.phat[((size_t)(ky * NKX + b / Z) * a.M + i) * N + z0 + b % Z] = v;
    });
}

template <int N, bool B = false, int V = 0>
__global__ void __launch_bounds__(512) ifft_xy32(StepArgs<float> a0, const StepArgs<float>* __restrict__ batch) {
    const StepArgs<float> a = pick_args<B>(a0, batch);
    constexpr int Z = XyShape<float, N, V>::Z, ZB = XyShape<float, N, V>::ZB;
    constexpr int NKX = N / 2 + 1, LS = NKX * Z, NR = N * N * N;
    using X = XLine<N, false>;
    constexpr int R = X::R, J = X::J;
    static_assert(X::ROW * (N / 2) % 2 == 0, "the half-spectrum buffer must stay 16-byte aligned");
    extern __shared__ __align__(16) unsigned char smem_raw[];
    float2* tw = reinterpret_cast<float2*>(smem_raw);
    float2* zb = tw + N;
    float2* out = zb + (size_t)ZB * (N / 2) * X::ROW;
    const int i = blockIdx.y, z0 = blockIdx.x * Z;
    for (int e = threadIdx.x; e < N; e += blockDim.x) tw[e] = a.twg[e];
    dep_wait<chained_step(N, 4, B)>();
    __syncthreads();
    // all loads issued up front: one Z-run (8 Z bytes) per (ky, kx)
    constexpr int CH = Z / 2;  // 16-byte chunks per run
    static_assert(Z % 2 == 0, "phat runs must be whole 16-byte chunks");
    for (int e = threadIdx.x; e < N * NKX * CH; e += blockDim.x) {
        const int col = e / CH, q = e % CH;
        cp_async16(out + (size_t)col * Z + 2 * q, a.phat + ((size_t)col * a.M + i) * N + z0 + 2 * q);
    }
    cp_async_wait_all();
    __syncthreads();
    fft_nat2perm<N, +1>(out, LS, LS, 1, tw);  // along y for every plane; row y now at perm_pos(y)
    for (int zz0 = 0; zz0 < Z; zz0 += ZB) {
        // Hermitian extension of rows (2p, 2p+1) packed as one complex row
        for (int w = threadIdx.x; w < ZB * (N / 2) * J; w += blockDim.x) {
            // plane fastest across the lanes, then j: neighbours in out
            const int q = w % ZB, j = w / ZB % J, p = w / (ZB * J), b = q * (N / 2) + p;
            const float2* ra = out + (size_t)perm_pos<N, float>(2 * p) * LS + zz0 + q;
            const float2* rb = out + (size_t)perm_pos<N, float>(2 * p + 1) * LS + zz0 + q;
            float2 v[R];
#pragma unroll
            for (int n = 0; n < R; ++n) v[n] = hermitian_pair<N>(ra, rb, n * J + j, Z);
            Dft<R>::template run<+1>(v);
            twiddles<R, +1>(v, j, tw);
            float2* row = zb + (size_t)b * X::ROW + j * X::S;
#pragma unroll
            for (int k = 0; k < R; ++k) row[k] = v[k];
        }
        __syncthreads();
        if (zz0 + ZB >= Z) dep_next<chained_step(N, 4, B)>();
        // packed row pair p holds rows 2p (real part) and 2p+1 (imaginary part)
        for (int w = threadIdx.x; w < ZB * (N / 2) * R; w += blockDim.x) {
            const int k = w % R, b = w / R;
            const float2* row = zb + (size_t)b * X::ROW + k;
            float2 v[J];
#pragma unroll
            for (int j = 0; j < J; ++j) v[j] = row[j * X::S];
            Dft<J>::template run<+1>(v);
            const size_t r = ((size_t)(z0 + zz0 + b / (N / 2)) * N + 2 * (b % (N / 2))) * N + k;
            float* dst = a.qout + (size_t)i * NR + r;
#pragma unroll
            for (int j = 0; j < J; ++j) {
                float2 u = cscale(v[j], a.minv);
                if (a.post) {  // split scheme: the second field half step
                    u.x *= a.post[r + R * j];
                    u.y *= a.post[r + R * j + N];
                }
                dst[R * j] = u.x;
                dst[R * j + N] = u.y;
            }
        }
        __syncthreads();
    }
}

// right-hand side only (init_pr test hook), out[i][r]
template <typename T, int N>
__global__ void __launch_bounds__(256) rhs_only(StepArgs<T> a, T* out) {
    constexpr int NR = N * N * N;
    const int64_t n = (int64_t)a.M * NR;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        out[e] = rhs_value<T, NR>(a, (size_t)e, (size_t)(e % NR));
}

// ------------------------------------------------------------ launchers
template <typename T> size_t smem_xy(int N, int variant) {
    using C = typename cvec<T>::t;
    const int z = xy_planes(N, sizeof(T), variant & 1), zb = (variant & 2) ? z : 1;
    const size_t plane = sizeof(T) == 8 ? (size_t)xplane(N) : (size_t)(N / 2) * xrow32_of(N);
    return sizeof(C) * ((size_t)N + zb * plane + (size_t)z * N * (N / 2 + 1)) +
           (sizeof(T) == 8 ? 2 * (size_t)xy_exps(N, z, zb) : 0);
}

// shared-memory limits of the pass A / pass C kernels of (T, N, B), once per
// (kernel, device); returns the first error
template <typename T, int N, bool B, int V> static const void* xy_kernel(bool do_a) {
    if constexpr (sizeof(T) == 4)
        return do_a ? (const void*)rhs_fft_xy32<N, B, V> : (const void*)ifft_xy32<N, B, V>;
    else
        return do_a ? (const void*)rhs_fft_xy<N, V> : (const void*)ifft_xy<N, V>;
}
constexpr int kXySmem = 220 * 1024;
template <typename T, int N, bool B> static cudaError_t set_xy_attrs() {
    cudaError_t e = cudaSuccess;
    auto set = [&](const void* a, const void* c) {
        for (const void* fn : {a, c}) {
            const cudaError_t r = smem_attr_once(fn, kXySmem);
            if (e == cudaSuccess) e = r;
        }
    };
    set(xy_kernel<T, N, B, 0>(true), xy_kernel<T, N, B, 0>(false));
    set(xy_kernel<T, N, B, 1>(true), xy_kernel<T, N, B, 1>(false));
    set(xy_kernel<T, N, B, 2>(true), xy_kernel<T, N, B, 2>(false));
    set(xy_kernel<T, N, B, 3>(true), xy_kernel<T, N, B, 3>(false));
    return e;
}

// Launch shape of passes A and C when none is set (threads = variant = 0), by
// the CTAs that fit an SM's shared memory: whole planes with all x-FFTs in one
// batched call (variant 2, the most work per barrier) with 256 threads while 4
// CTAs fit, else half planes and one plane's x-FFTs at a time (variant 1, the
// smallest CTAs), with 512 threads where few of those fit.  Measured (us per
// step, the next best of the other seven shapes in brackets): FP32 pass A 24^3
// 11.1 (12.3), 48^3 53.8 (54.3), 64^3 147 (143, but 4 more in pass C), 96^3 436
// (507); pass C 40^3 18.9 (20.9), 64^3 88.6 (90.2), 96^3 228 (247); FP64 pass
// A 40^3 112 (120), 64^3 527 (655); pass C 24^3 14.6 (18.7).
template <typename T> static void xy_shape(int N, int& threads, int& variant) {
    if (threads == 0 && variant == 0) {
        auto ctas = [&](int v) { return (int)(227 * 1024 / (smem_xy<T>(N, v) + 1024)); };
        variant = ctas(2) >= 4 ? 2 : 1;
        threads = variant == 2 || ctas(1) >= (sizeof(T) == 4 ? 5 : 2) ? 256 : 512;
    }
    threads = threads == 512 ? 512 : 256;
}

// generic pass A / pass C launches in variant V (bit 0 half planes, bit 1
// batched x-FFTs)
template <typename T, int N, bool B, int V>
static void launch_xy(bool do_a, const StepArgs<T>& a, const StepArgs<T>* batch, int M, int count, int threads,
                      bool chain, cudaStream_t st) {
    constexpr int Z = XyShape<T, N, V>::Z;
    const size_t sxy = smem_xy<T>(N, V);
    const dim3 g(N / Z, M, count);
    if constexpr (sizeof(T) == 4) {
        if (do_a)
            launch_chained(chain && chained_step(N, 4, B), rhs_fft_xy32<N, B, V>, g, threads, sxy, st, a, batch);
        else
            launch_chained(chain && chained_step(N, 4, B), ifft_xy32<N, B, V>, g, threads, sxy, st, a, batch);
    } else {
        if (do_a)
            launch_chained(chain && chained_step(N, 8, B), rhs_fft_xy<N, V>, g, threads, sxy, st, a);
        else
            launch_chained(chain && chained_step(N, 8, B), ifft_xy<N, V>, g, threads, sxy, st, a);
    }
}

template <typename T, int N, bool B>
static void launch_xy_any(int variant, bool do_a, const StepArgs<T>& a, const StepArgs<T>* batch, int M, int count,
                          int threads, bool chain, cudaStream_t st) {
    xy_shape<T>(N, threads, variant);
    if ((variant & 2) && smem_xy<T>(N, variant) > kXySmem) variant &= 1;  // batched x-FFTs do not fit
    switch (variant & 3) {
        case 1: launch_xy<T, N, B, 1>(do_a, a, batch, M, count, threads, chain, st); break;
        case 2: launch_xy<T, N, B, 2>(do_a, a, batch, M, count, threads, chain, st); break;
        case 3: launch_xy<T, N, B, 3>(do_a, a, batch, M, count, threads, chain, st); break;
        default: launch_xy<T, N, B, 0>(do_a, a, batch, M, count, threads, chain, st); break;
    }
}

template <typename T, int N> static cudaError_t launch_n(const StepLaunch<T>& s, cudaStream_t st) {
    if (const cudaError_t ea = set_xy_attrs<T, N, false>(); ea != cudaSuccess) return ea;
    if (s.events) cudaEventRecord(s.events[0], st);
    if (s.do_a) launch_xy_any<T, N, false>(s.xy_z, true, s.step, nullptr, s.step.M, 1, s.xy_threads, s.chain_a, st);
    if (s.events) cudaEventRecord(s.events[1], st);
    if (s.do_b) launch_solve<T>(N, s.solve, st, s.solve_threads);
    if (s.events) cudaEventRecord(s.events[2], st);
    if (s.do_c) launch_xy_any<T, N, false>(s.xy_z, false, s.step, nullptr, s.step.M, 1, s.xy_threads, true, st);
    if (s.events) cudaEventRecord(s.events[3], st);
    return cudaGetLastError();
}

template <int N> static cudaError_t launch_batched_n(const BatchLaunch<float>& b, cudaStream_t st) {
    if (const cudaError_t ea = set_xy_attrs<float, N, true>(); ea != cudaSuccess) return ea;
    launch_xy_any<float, N, true>(b.xy_z, true, StepArgs<float>{}, b.dstep, b.M, b.count, b.xy_threads, false, st);
    cudaError_t e = launch_solve_batched(N, b, st);
    if (e != cudaSuccess) return e;
    launch_xy_any<float, N, true>(b.xy_z, false, StepArgs<float>{}, b.dstep, b.M, b.count, b.xy_threads, false, st);
    return cudaGetLastError();
}

cudaError_t launch_step_batched(int N, const BatchLaunch<float>& b, cudaStream_t st) {
    switch (N) {
#define WLC_CASE(n) \
    case n:         \
        return launch_batched_n<n>(b, st);
        WLC_FOR_EACH_BATCH_N(WLC_CASE)
#undef WLC_CASE
        default:
            return cudaErrorInvalidValue;
    }
}

// function attributes of the batched kernels, set outside any stream capture
cudaError_t prepare_step_batched(int N) {
    switch (N) {
#define WLC_CASE(n)                                                       \
    case n: {                                                             \
        const cudaError_t ea = set_xy_attrs<float, n, true>();            \
        return ea != cudaSuccess ? ea : prepare_solve_batched(n);         \
    }
        WLC_FOR_EACH_BATCH_N(WLC_CASE)
#undef WLC_CASE
        default:
            return cudaErrorInvalidValue;
    }
}

template <typename T> cudaError_t launch_step(int N, const StepLaunch<T>& s, cudaStream_t st) {
    switch (N) {
#define WLC_CASE(n) \
    case n:         \
        return launch_n<T, n>(s, st);
        WLC_FOR_EACH_N(WLC_CASE)
#undef WLC_CASE
        default:
            return cudaErrorInvalidValue;
    }
}

template <typename T> cudaError_t launch_rhs_only(int N, const StepArgs<T>& a, T* out, cudaStream_t st) {
    switch (N) {
#define WLC_CASE(n)                                                                \
    case n: {                                                                      \
        const int64_t tot = (int64_t)a.M * n * n * n;                              \
        const int g = (int)((tot + 255) / 256 > 4096 ? 4096 : (tot + 255) / 256); \
        rhs_only<T, n><<<g, 256, 0, st>>>(a, out);                                 \
        return cudaGetLastError();                                                 \
    }
        WLC_FOR_EACH_N(WLC_CASE)
#undef WLC_CASE
        default:
            return cudaErrorInvalidValue;
    }
}

template cudaError_t launch_rhs_only<double>(int, const StepArgs<double>&, double*, cudaStream_t);
template cudaError_t launch_rhs_only<float>(int, const StepArgs<float>&, float*, cudaStream_t);
template cudaError_t launch_step<double>(int, const StepLaunch<double>&, cudaStream_t);
template cudaError_t launch_step<float>(int, const StepLaunch<float>&, cudaStream_t);
template size_t smem_xy<double>(int, int);
template size_t smem_xy<float>(int, int);

}  // namespace wlc
