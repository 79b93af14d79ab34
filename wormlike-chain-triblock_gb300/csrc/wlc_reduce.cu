// wlc_reduce.cu -- layout conversion, field preprocessing, density / Q /
// orientation tensor / free energy kernels.
//
// Reference: density() SCFT_Density_FE_ABC.f90:3-271 (per-block
// restatement), SCFT_Density_FE.f90:48-220 (AB form), free_energy()
// SCFT_Density_FE.f90:273-342, integrators utility_mod.f90:195-374,
// Sum_sparse_2D utility_mod.f90:376-407.
//
// All reductions are deterministic: fixed partition per CTA, fixed-order
// tree in shared memory, one final CTA summing the partials in order.
#include <algorithm>
#include <cstdint>

#include "wlc_attr.h"
#include "wlc_reduce.h"

namespace wlc {

// ------------------------------------------------------------ layouts
// reference layout [r][i] (coefficient fastest) <-> internal [i][r]
template <typename T>
__global__ void to_internal(const double* __restrict__ ref, T* __restrict__ out, int M, int64_t nr) {
    __shared__ double tile[32][33];
    const int64_t r0 = (int64_t)blockIdx.x * 32;
    const int i0 = blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int64_t r = r0 + k;
        const int i = i0 + threadIdx.x;
        if (r < nr && i < M) tile[k][threadIdx.x] = ref[r * M + i];
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int i = i0 + k;
        const int64_t r = r0 + threadIdx.x;
        if (r < nr && i < M) out[(int64_t)i * nr + r] = (T)tile[threadIdx.x][k];
    }
}

template <typename T>
__global__ void to_reference(const T* __restrict__ in, double* __restrict__ ref, int M, int64_t nr) {
    __shared__ double tile[32][33];
    const int64_t r0 = (int64_t)blockIdx.x * 32;
    const int i0 = blockIdx.y * 32;
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int i = i0 + k;
        const int64_t r = r0 + threadIdx.x;
        if (r < nr && i < M) tile[k][threadIdx.x] = (double)in[(int64_t)i * nr + r];
    }
    __syncthreads();
    for (int k = threadIdx.y; k < 32; k += blockDim.y) {
        const int64_t r = r0 + k;
        const int i = i0 + threadIdx.x;
        if (r < nr && i < M) ref[r * M + i] = tile[threadIdx.x][k];
    }
}

// q(0) = delta_{i0} (MDE_ABC.f90:40-45, :62-67)
template <typename T> __global__ void set_delta(T* q, int M, int64_t nr) {
    const int64_t n = (int64_t)M * nr;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        q[e] = e < nr ? (T)1 : (T)0;
}

// order-3 history coefficients per block: cf[blk][3][nr] =
// (3 - 3 ds w, -3/2 + 3 ds w, third - ds w); then dsw[blk][nr] = ds w at
// cf + 9 nr and the split scheme's field half-step factors e^{-w ds/2} at
// cf + 12 nr (split_operator_MDE_mod.f90:163-166)
template <typename T>
__global__ void make_cf(const double* __restrict__ w, T* __restrict__ cf, double ds, double third, int64_t nr) {
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nr; r += (int64_t)gridDim.x * blockDim.x)
        for (int b = 0; b < 3; ++b) {
            const double W = w[b * nr + r];
            T* o = cf + (size_t)b * 3 * nr;
            o[r] = (T)(3.0 - 3.0 * ds * W);
            o[nr + r] = (T)(-1.5 + 3.0 * ds * W);
            o[2 * nr + r] = (T)(third - ds * W);
            cf[(size_t)(9 + b) * nr + r] = (T)(ds * W);
            cf[(size_t)(12 + b) * nr + r] = (T)exp(-0.5 * ds * W);
        }
}

// Maier-Saupe term ds * sum_j Theta_ij(r) h_j(r), h the BDF history
// combination of the given order (calc_THETAij and the Theta loop of
// init_pr, wormlike_MDE_2dcomp_mod.f90:5-110, MDE_ABC.f90:256-268).
// 16-byte vector access of 16/sizeof(T) consecutive values (16-byte aligned)
template <typename T> struct VecOf;
template <> struct VecOf<float> { using t = float4; };
template <> struct VecOf<double> { using t = double2; };
template <typename T> __device__ __forceinline__ void vload(const T* p, T* v) {
    const typename VecOf<T>::t x = *reinterpret_cast<const typename VecOf<T>::t*>(p);
    if constexpr (sizeof(T) == 4) {
        v[0] = x.x;
        v[1] = x.y;
        v[2] = x.z;
        v[3] = x.w;
    } else {
        v[0] = x.x;
        v[1] = x.y;
    }
}
template <typename T> __device__ __forceinline__ void vstore(T* p, const T* v) {
    typename VecOf<T>::t x;
    if constexpr (sizeof(T) == 4) {
        x.x = v[0];
        x.y = v[1];
        x.z = v[2];
        x.w = v[3];
    } else {
        x.x = v[0];
        x.y = v[1];
    }
    *reinterpret_cast<typename VecOf<T>::t*>(p) = x;
}

// ------------------------------------------------------------ coupling lists
// The per-point kernels below (Theta term, orientation tensor) are sparse
// products with the coefficient vector of every grid point.  One CTA stages
// the lists once and walks tiles of TILE points; a thread takes P points (one
// 16-byte vector) and every kGroups-th row, longest rows first, so that one
// list entry (two broadcast reads) and one 16-byte read of the tile serve P
// points.  A component's entries of a row are summed before the point's
// factor is applied: one multiply-add per entry and point.
constexpr int kGroups = 16;
template <typename T> struct Pts {
    static constexpr int P = 16 / sizeof(T), LANES = PointTile<T>::value / P, THREADS = LANES * kGroups;
};

template <typename T> struct ListSmem {
    T *val, *gval;
    uint16_t *ptr, *gptr;
    int16_t *col, *gcol, *order;
};
template <typename T> __host__ __device__ inline size_t list_bytes(int n, int ng, int M) {
    return sizeof(T) * ((size_t)n + 5 * ng) + 2 * ((size_t)5 * M + 1 + M + 1 + n + ng + M);
}
template <typename T> __device__ __forceinline__ ListSmem<T> stage_lists(const ClassLists& l, int M, void* at) {
    ListSmem<T> m;
    m.val = reinterpret_cast<T*>(at);
    m.gval = m.val + l.n;
    m.ptr = reinterpret_cast<uint16_t*>(m.gval + 5 * l.ng);
    m.gptr = m.ptr + 5 * M + 1;
    m.col = reinterpret_cast<int16_t*>(m.gptr + M + 1);
    m.gcol = m.col + l.n;
    m.order = m.gcol + l.ng;
    for (int e = threadIdx.x; e < l.n; e += blockDim.x) {
        m.val[e] = (T)l.val[e];
        m.col[e] = l.col[e];
    }
    for (int e = threadIdx.x; e < 5 * l.ng; e += blockDim.x) m.gval[e] = (T)l.gval[e];
    for (int e = threadIdx.x; e < l.ng; e += blockDim.x) m.gcol[e] = l.gcol[e];
    for (int e = threadIdx.x; e <= 5 * M; e += blockDim.x) m.ptr[e] = l.ptr[e];
    for (int e = threadIdx.x; e <= M; e += blockDim.x) m.gptr[e] = l.gptr[e];
    for (int e = threadIdx.x; e < M; e += blockDim.x) m.order[e] = l.order[e];
    return m;
}

// sum of the entries [e0, e1) times the tile's coefficients, at P points
template <typename T>
__device__ __forceinline__ void gather_sum(const ListSmem<T>& m, int e0, int e1, const T* tile, T* y) {
    constexpr int P = Pts<T>::P, TILE = PointTile<T>::value;
#pragma unroll
    for (int u = 0; u < P; ++u) y[u] = (T)0;
#pragma unroll 2
    for (int e = e0; e < e1; ++e) {
        const T v = m.val[e];
        T h[P];
        vload<T>(tile + m.col[e] * TILE, h);
#pragma unroll
        for (int u = 0; u < P; ++u) y[u] = fma(v, h[u], y[u]);
    }
}

// shared-memory layout of ms_term: hc[M][TILE] | coef[5][TILE] | lists
template <typename T> __host__ __device__ inline size_t ms_smem_bytes(const ClassLists& tl, int M) {
    return sizeof(T) * (size_t)(M + 5) * PointTile<T>::value + list_bytes<T>(tl.n, tl.ng, M);
}

// Bound by the shared-memory reads of the tile (one 16-byte read per entry and
// P points).  128^3, L = 12 in FP32: 6.1 ms a launch with one point a thread
// and all five components of every entry, 2.5 ms in this form.
template <typename T>
__global__ void __launch_bounds__(Pts<T>::THREADS)
    ms_term(const T* __restrict__ h1, const T* __restrict__ h2, const T* __restrict__ h3, int order,
            const double* __restrict__ mop, ClassLists tl, double ds, double thresh, int M, int64_t nr,
            T* __restrict__ out) {
    constexpr int TILE = PointTile<T>::value, P = Pts<T>::P;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* hc = reinterpret_cast<T*>(smem_raw);  // [M][TILE]: BDF history combination of the tile's points
    T* sco = hc + (size_t)M * TILE;          // [5][TILE]: factors of the components
    const ListSmem<T> m = stage_lists<T>(tl, M, sco + 5 * TILE);
    const int k = (threadIdx.x % Pts<T>::LANES) * P, g = threadIdx.x / Pts<T>::LANES;
    const T th_min = (T)thresh;
    for (int64_t r0 = (int64_t)blockIdx.x * TILE; r0 < nr; r0 += (int64_t)gridDim.x * TILE) {
        __syncthreads();  // lists staged / previous tile consumed
        for (int idx = threadIdx.x; idx < M * (TILE / P); idx += blockDim.x) {
            const int j = idx / (TILE / P), kk = (idx % (TILE / P)) * P;
            const int64_t o = (int64_t)j * nr + r0 + kk;  // nr is a multiple of TILE
            T v[P], q1[P], q2[P], q3[P];
            vload<T>(h1 + o, q1);
            if (order >= 2) vload<T>(h2 + o, q2);
            if (order >= 3) vload<T>(h3 + o, q3);
#pragma unroll
            for (int u = 0; u < P; ++u) {
                if (order == 1)
                    v[u] = q1[u];
                else if (order == 2)
                    v[u] = (T)2 * q1[u] - q2[u];
                else
                    v[u] = (T)3 * q1[u] - (T)3 * q2[u] + q3[u];
            }
            vstore<T>(hc + j * TILE + kk, v);
        }
        // Theta_ij(r) = sum_c coef_c T_c(i,j)
        // (M01 = mop[0 + 3*1] = M_OP(k,0,1) in Fortran order; the tensor is symmetric)
        for (int idx = threadIdx.x; idx < 5 * TILE; idx += blockDim.x) {
            const int c = idx / TILE;
            const int64_t r = r0 + idx % TILE;
            const double v = c == 0   ? mop[r] - mop[4 * nr + r]
                             : c == 1 ? mop[8 * nr + r]
                                      : mop[(c == 2 ? 3 : c == 3 ? 6 : 7) * nr + r];
            sco[idx] = (T)v;
        }
        __syncthreads();
        // entries with |Theta| below the threshold are dropped: none or all of
        // a component's where its factor is large or tiny enough, else entry
        // by entry (bit c of mixed)
        T cf[5][P];
        unsigned mixed = 0;
#pragma unroll
        for (int c = 0; c < 5; ++c) {
            vload<T>(sco + c * TILE + k, cf[c]);
#pragma unroll
            for (int u = 0; u < P; ++u) {
                const T a = fabs(cf[c][u]);
                if (a * (T)tl.vmax[c] < th_min * (T)0.5)
                    cf[c][u] = (T)0;
                else if (!(a * (T)tl.vmin[c] > th_min * (T)2))
                    mixed |= 1u << c;
            }
        }
        for (int row = g; row < M; row += kGroups) {
            const int i = m.order[row];
            const uint16_t* pt = m.ptr + 5 * i;
            T acc[P] = {};
            int e0 = pt[0];
#pragma unroll
            for (int c = 0; c < 5; ++c) {
                const int e1 = pt[c + 1];
                if (!((mixed >> c) & 1u)) {
                    T y[P];
                    gather_sum<T>(m, e0, e1, hc + k, y);
#pragma unroll
                    for (int u = 0; u < P; ++u) acc[u] = fma(cf[c][u], y[u], acc[u]);
                } else {
                    for (int e = e0; e < e1; ++e) {
                        const T v = m.val[e];
                        T h[P];
                        vload<T>(hc + m.col[e] * TILE + k, h);
#pragma unroll
                        for (int u = 0; u < P; ++u) {
                            const T th = cf[c][u] * v;
                            if (!(fabs(th) < th_min)) acc[u] = fma(th, h[u], acc[u]);
                        }
                    }
                }
                e0 = e1;
            }
            for (int e = m.gptr[i]; e < m.gptr[i + 1]; ++e) {
                T h[P];
                vload<T>(hc + m.gcol[e] * TILE + k, h);
#pragma unroll
                for (int u = 0; u < P; ++u) {
                    T th = (T)0;
#pragma unroll
                    for (int c = 0; c < 5; ++c) th = fma(sco[c * TILE + k + u], m.gval[5 * e + c], th);
                    if (!(fabs(th) < th_min)) acc[u] = fma(th, h[u], acc[u]);
                }
            }
#pragma unroll
            for (int u = 0; u < P; ++u) acc[u] *= (T)ds;
            vstore<T>(out + (int64_t)i * nr + r0 + k, acc);
        }
    }
}

// ------------------------------------------------------------ densities
// Running dot products in (at least) FP64 accuracy at P points.  FP32 slices:
// a product and its error are exact in two floats and are added to a sum of
// three floats by error-free additions (72 bits; the FP64 pipe has 1/64 of
// the FP32 rate, and one multiply-add with its two conversions costs 192
// clocks of a scheduler there against 26 here).  That holds while the largest
// product lies within 2^-90 .. 2^100: errors of smaller products, below 2^-149,
// are then under 2^-59 of it and no sum overflows; or while one factor is zero
// throughout (most coefficients at the chain's ends).  Otherwise holds() is
// false and dot_fp64 sums again in FP64.
__device__ __forceinline__ float two_sum(float a, float b, float& err) {
    const float s = __fadd_rn(a, b), bb = __fsub_rn(s, a);
    err = __fadd_rn(__fsub_rn(a, __fsub_rn(s, bb)), __fsub_rn(b, bb));
    return s;
}
// sum over the rows first, first + step, ... < M (through order, if given) of a c
static __device__ __noinline__ double dot_fp64(const float* a, const float* c, const int16_t* order, int first, int step,
                                               int M, int64_t nr) {
    double s = 0.0;
    for (int row = first; row < M; row += step) {
        const int64_t o = (order ? order[row] : row) * nr;
        s = fma((double)a[o], (double)c[o], s);
    }
    return s;
}
// FP64 slices: K sums of every K-th product (add's k), so that a long row of
// coefficients is not one chain of roundings
template <typename T, int P, int K = 1> struct Dots;
template <int P, int K> struct Dots<double, P, K> {
    static constexpr int W = 1;  // words per point
    double s[K][P] = {};
    __device__ __forceinline__ void add(int u, double a, double b, int k = 0) { s[k][u] = fma(a, b, s[k][u]); }
    __device__ __forceinline__ double get(int u) const {
        if constexpr (K == 4) return (s[0][u] + s[1][u]) + (s[2][u] + s[3][u]);
        return s[0][u];
    }
};
template <int P, int K> struct Dots<float, P, K> {
    static constexpr int W = 3;
    float s[P] = {}, c[P] = {}, d[P] = {}, top[P] = {};  // top: largest product
    unsigned abits = 0, bbits = 0;                       // bits set in any factor, at any point
    __device__ __forceinline__ void add3(int u, float p, float e, float f) {
        float t1, t2, t3;
        s[u] = two_sum(s[u], p, t1);
        c[u] = two_sum(c[u], t1, t2);
        c[u] = two_sum(c[u], e, t3);
        d[u] = __fadd_rn(d[u], __fadd_rn(__fadd_rn(t2, t3), f));
    }
    __device__ __forceinline__ void add(int u, float a, float b, int = 0) {
        const float p = __fmul_rn(a, b);
        top[u] = fmaxf(top[u], fabsf(p));
        abits |= __float_as_uint(a);
        bbits |= __float_as_uint(b);
        add3(u, p, __fmaf_rn(a, b, -p), 0.0f);
    }
    __device__ __forceinline__ bool holds(int u) const {
        const bool zero = abits << 1 == 0 || bbits << 1 == 0;
        return s[u] == s[u] && (zero || (top[u] >= 0x1p-90f && top[u] <= 0x1p100f));
    }
    __device__ __forceinline__ double get(int u) const { return (double)s[u] + ((double)c[u] + (double)d[u]); }
};

// raw[b][r] = sum_i S1_{s in block b}(q_i q*_i); junc[j][r] = sum_i q_i q*_i at
// s = NA, NA+NB, Nmax; qend[r] = q_0(r, Nmax).  Every slice is read once.  A
// CTA's threads are G groups of coefficients for 256 / G times P points; the
// larger G serves grids that would not fill the SMs otherwise.
// 64^3, L = 10, 101 slices, four rows of loads in flight: FP32 (25.6 GB) 5.6 ms
// (8.0 row by row; with conversions and multiply-adds on the FP64 pipe 10.7
// more), FP64 7.1 ms (7.2).
template <typename T, int P, int G>
__global__ void __launch_bounds__(256)
    density_accum(const T* __restrict__ qf, const T* __restrict__ qb, DensityArgs d, double* __restrict__ raw,
                  double* __restrict__ junc, double* __restrict__ qend) {
    constexpr int LANES = 256 / G;
    __shared__ double red[G > 1 ? G : 1][G > 1 ? LANES * P : 1];
    const int64_t nr = d.nr, sl = (int64_t)d.M * nr;
    const int lane = threadIdx.x % LANES, g = threadIdx.x / LANES;
    const int64_t r = ((int64_t)blockIdx.x * LANES + lane) * P;
    const bool in = r < nr;
    double acc[3][P] = {};
    // sum over the groups of v[], for the threads of group 0
    auto over_groups = [&](double* v) {
        if constexpr (G > 1) {
            __syncthreads();
#pragma unroll
            for (int u = 0; u < P; ++u) red[g][lane * P + u] = v[u];
            __syncthreads();
            if (g == 0)
#pragma unroll
                for (int u = 0; u < P; ++u) {
                    v[u] = red[0][lane * P + u];
                    for (int q = 1; q < G; ++q) v[u] += red[q][lane * P + u];
                }
        }
    };
    const int sj[3] = {d.nstart[1], d.nstart[2], d.nmax};
    for (int s = 0; s <= d.nmax; ++s) {
        Dots<T, P, 4> dot;
        if (in) {
            const T* a = qf + s * sl + r;
            const T* c = qb + s * sl + r;
            auto row = [&](int i, int k) {
                T x[P], y[P];
                if constexpr (P > 1) {
                    vload<T>(a + i * nr, x);
                    vload<T>(c + i * nr, y);
                } else {
                    x[0] = a[i * nr];
                    y[0] = c[i * nr];
                }
#pragma unroll
                for (int u = 0; u < P; ++u) dot.add(u, x[u], y[u], k);
            };
            int i = g;
            for (; i + 3 * G < d.M; i += 4 * G) {
#pragma unroll
                for (int k = 0; k < 4; ++k) row(i + k * G, k);
            }
            for (; i < d.M; i += G) row(i, 0);
        }
        double v[P];
#pragma unroll
        for (int u = 0; u < P; ++u) {
            v[u] = dot.get(u);
            if constexpr (sizeof(T) == 4)
                if (in && !dot.holds(u)) v[u] = dot_fp64(qf + s * sl + r + u, qb + s * sl + r + u, nullptr, g, G, d.M, nr);
        }
        for (int b = 0; b < 3; ++b) {
            const int j = s - d.nstart[b], n = d.ns[b];
            if (n <= 0 || j < 0 || j > n) continue;
            const double wgt = (j == 0 || j == n) ? 1.0 : ((j & 1) ? 4.0 : 2.0);
#pragma unroll
            for (int u = 0; u < P; ++u) acc[b][u] += wgt * v[u];
        }
        if (s == sj[0] || s == sj[1] || s == sj[2]) {
            over_groups(v);
            if (g == 0 && in)
                for (int j = 0; j < 3; ++j)
                    if (s == sj[j])
#pragma unroll
                        for (int u = 0; u < P; ++u) junc[j * nr + r + u] = v[u];
        }
    }
    for (int b = 0; b < 3; ++b) {
        over_groups(acc[b]);
        if (g == 0 && in)
#pragma unroll
            for (int u = 0; u < P; ++u) raw[b * nr + r + u] = acc[b][u] * (d.ds / 3.0);
    }
    if (g == 0 && in)
#pragma unroll
        for (int u = 0; u < P; ++u) qend[r + u] = (double)qf[(int64_t)d.nmax * sl + r + u];
}

// shared-memory layout of the tiled density / tensor kernels: the tile of q*
// [M][TILE], with the groups' partial sums over it [kGroups][W + 5][TILE]
// afterwards | lists (with the tensor)
template <typename T> __host__ __device__ inline size_t slice_tile_bytes(int M, bool want_s) {
    const size_t red = sizeof(T) * (size_t)kGroups * (Dots<T, 1>::W + 5) * PointTile<T>::value;
    const size_t tile = want_s ? sizeof(T) * (size_t)M * PointTile<T>::value : 0;
    return red > tile ? red : tile;
}
template <typename T> __host__ __device__ inline size_t slice_smem_bytes(const ClassLists& jl, int M, bool want_s) {
    return slice_tile_bytes<T>(M, want_s) + (want_s ? list_bytes<T>(jl.n, jl.ng, M) : 0);
}

// Sums of one slice at the tile's points: sum_i q_i q*_i (FP64 accuracy) and,
// with the lists, the five forms q^T J_t q*.  Called by the whole CTA; the
// partial sums over the groups of rows end in red.
template <typename T>
__device__ __forceinline__ void slice_sums(const T* __restrict__ a, const T* __restrict__ c, int M, int64_t nr, int64_t r0,
                                           const ListSmem<T>* lists, T* tile) {
    constexpr int TILE = PointTile<T>::value, P = Pts<T>::P, W = Dots<T, 1>::W;
    const int k = (threadIdx.x % Pts<T>::LANES) * P, g = threadIdx.x / Pts<T>::LANES;
    Dots<T, P> dot;
    T f[5][P] = {};
    if (lists) {
        for (int idx = threadIdx.x; idx < M * (TILE / P); idx += blockDim.x) {
            const int i = idx / (TILE / P), kk = (idx % (TILE / P)) * P;
            T v[P];
            vload<T>(c + (int64_t)i * nr + r0 + kk, v);
            vstore<T>(tile + i * TILE + kk, v);
        }
        __syncthreads();
        for (int row = g; row < M; row += kGroups) {
            const int i = lists->order[row];
            T q[P], p[P];
            vload<T>(a + (int64_t)i * nr + r0 + k, q);
            vload<T>(tile + i * TILE + k, p);
#pragma unroll
            for (int u = 0; u < P; ++u) dot.add(u, q[u], p[u]);
            const uint16_t* pt = lists->ptr + 5 * i;
            int e0 = pt[0];
#pragma unroll
            for (int t = 0; t < 5; ++t) {
                const int e1 = pt[t + 1];
                T y[P];
                gather_sum<T>(*lists, e0, e1, tile + k, y);
#pragma unroll
                for (int u = 0; u < P; ++u) f[t][u] = fma(q[u], y[u], f[t][u]);
                e0 = e1;
            }
        }
        __syncthreads();  // the tile becomes the space of the partial sums
    } else {
#pragma unroll 4
        for (int i = g; i < M; i += kGroups) {
            T q[P], p[P];
            vload<T>(a + (int64_t)i * nr + r0 + k, q);
            vload<T>(c + (int64_t)i * nr + r0 + k, p);
#pragma unroll
            for (int u = 0; u < P; ++u) dot.add(u, q[u], p[u]);
        }
    }
    T* red = tile + (size_t)g * (W + 5) * TILE + k;
#pragma unroll
    for (int u = 0; u < P; ++u) {
        if constexpr (sizeof(T) == 8) {
            red[u] = dot.get(u);
        } else {  // the three words of the sum, or the two of an FP64 sum and a not-a-number
            red[u] = dot.s[u];
            red[TILE + u] = dot.c[u];
            red[2 * TILE + u] = dot.d[u];
            if (!dot.holds(u)) {
                const int64_t o = r0 + k + u;
                const double v = dot_fp64(a + o, c + o, lists ? lists->order : nullptr, g, kGroups, M, nr);
                red[u] = __int_as_float(__double2hiint(v));
                red[TILE + u] = __int_as_float(__double2loint(v));
                red[2 * TILE + u] = __int_as_float(0x7fc00000);
            }
        }
        if (lists)
#pragma unroll
            for (int t = 0; t < 5; ++t) red[(W + t) * TILE + u] = f[t][u];
    }
    __syncthreads();
}
// the tile's point k: the dot product, and tensor component t
template <typename T> __device__ __forceinline__ double slice_dot(const T* red, int k) {
    constexpr int TILE = PointTile<T>::value, W = Dots<T, 1>::W;
    double x = 0.0;
    Dots<T, 1> dot;
    for (int g = 0; g < kGroups; ++g) {
        const T* w = red + (size_t)g * (W + 5) * TILE + k;
        if constexpr (sizeof(T) == 8) {
            x += w[0];
        } else {
            const float d = w[2 * TILE];
            if (d == d)
                dot.add3(0, w[0], w[TILE], d);
            else
                x += __hiloint2double(__float_as_int(w[0]), __float_as_int(w[TILE]));
        }
    }
    return dot.get(0) + x;
}
template <typename T> __device__ __forceinline__ double slice_form(const T* red, int t, int k) {
    constexpr int TILE = PointTile<T>::value, W = Dots<T, 1>::W;
    T x = (T)0, y = (T)0;  // component t; J11, J22: half sum and half difference
    const int ta = t < 2 ? 0 : t;
    for (int g = 0; g < kGroups; ++g) {
        const T* w = red + ((size_t)g * (W + 5) + W) * TILE + k;
        x += w[ta * TILE];
        if (t < 2) y += w[TILE];
    }
    return (double)(t == 0 ? x + y : t == 1 ? x - y : x);
}

// orientation tensor per block (SCFT_Density_FE.f90:161-220):
// sraw[b][t][r] = S1_s( q^T J_t q* ), t = 11, 22, 12, 13, 23
template <typename T>
__global__ void __launch_bounds__(Pts<T>::THREADS)
    stensor_accum(const T* __restrict__ qf, const T* __restrict__ qb, DensityArgs d, ClassLists jl,
                  double* __restrict__ sraw) {
    constexpr int TILE = PointTile<T>::value, NT = Pts<T>::THREADS, Q = (5 * TILE + NT - 1) / NT;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* tile = reinterpret_cast<T*>(smem_raw);
    const ListSmem<T> m = stage_lists<T>(jl, d.M, smem_raw + slice_tile_bytes<T>(d.M, true));
    const int64_t nr = d.nr, sl = (int64_t)d.M * nr, r0 = (int64_t)blockIdx.x * TILE;
    double acc[Q][3] = {};
    for (int s = 0; s <= d.nmax; ++s) {
        __syncthreads();  // lists staged / sums of the previous slice read
        slice_sums<T>(qf + s * sl, qb + s * sl, d.M, nr, r0, &m, tile);
#pragma unroll
        for (int q = 0; q < Q; ++q) {
            const int idx = threadIdx.x + q * NT;
            if (idx >= 5 * TILE) break;
            const double v = slice_form<T>(tile, idx / TILE, idx % TILE);
#pragma unroll
            for (int b = 0; b < 3; ++b) {
                const int j = s - d.nstart[b], n = d.ns[b];
                if (n <= 0 || j < 0 || j > n) continue;
                acc[q][b] += ((j == 0 || j == n) ? 1.0 : ((j & 1) ? 4.0 : 2.0)) * v;
            }
        }
    }
#pragma unroll
    for (int q = 0; q < Q; ++q) {
        const int idx = threadIdx.x + q * NT;
        if (idx >= 5 * TILE) break;
#pragma unroll
        for (int b = 0; b < 3; ++b)
            sraw[((int64_t)b * 5 + idx / TILE) * nr + r0 + idx % TILE] = acc[q][b] * d.ds / 3.0;
    }
}

// Streamed form of density_accum / stensor_accum: one slice s per launch,
// issued by the backward sweep right after q*(s) is computed (descending s),
// so the q* slices need not be stored.  Same Simpson weights per block.  One
// CTA walks tiles of TILE points of one instance.
// 128^3, L = 12 with the tensor in FP32: 9.9 -> 2.5 ms a launch (2.4 without the
// guard of the sums' range).
template <typename T>
__device__ __forceinline__ void density_slice_tiles(const T* __restrict__ a, const T* __restrict__ c,
                                                    const DensityArgs& d, int s, int want_s, const ClassLists& jl,
                                                    double* __restrict__ raw, double* __restrict__ junc,
                                                    double* __restrict__ qend, double* __restrict__ sraw) {
    constexpr int TILE = PointTile<T>::value;
    extern __shared__ __align__(16) unsigned char smem_raw[];
    T* tile = reinterpret_cast<T*>(smem_raw);
    ListSmem<T> m{};
    if (want_s) m = stage_lists<T>(jl, d.M, smem_raw + slice_tile_bytes<T>(d.M, true));
    const int64_t nr = d.nr;
    double wgt[3];
    for (int b = 0; b < 3; ++b) {
        const int j = s - d.nstart[b], n = d.ns[b];
        wgt[b] = (n > 0 && j >= 0 && j <= n) ? ((j == 0 || j == n) ? 1.0 : ((j & 1) ? 4.0 : 2.0)) : 0.0;
    }
    const int sj[3] = {d.nstart[1], d.nstart[2], d.nmax};
    const double scl = d.ds / 3.0;
    for (int64_t r0 = (int64_t)blockIdx.x * TILE; r0 < nr; r0 += (int64_t)gridDim.x * TILE) {
        __syncthreads();  // lists staged / previous tile's sums read
        slice_sums<T>(a, c, d.M, nr, r0, want_s ? &m : nullptr, tile);
        for (int idx = threadIdx.x; idx < (want_s ? 6 : 1) * TILE; idx += blockDim.x) {
            const int t = idx / TILE - 1, k = idx % TILE;
            const int64_t r = r0 + k;
            if (t < 0) {
                const double sum = slice_dot<T>(tile, k);
                for (int b = 0; b < 3; ++b)
                    if (wgt[b] != 0.0) raw[b * nr + r] += wgt[b] * sum;
                for (int j = 0; j < 3; ++j)
                    if (s == sj[j]) junc[j * nr + r] = sum;
                if (s == d.nmax) qend[r] = (double)a[r];
                if (s == 0)  // last slice of the backward sweep
                    for (int b = 0; b < 3; ++b) raw[b * nr + r] *= scl;
            } else {
                const double st = slice_form<T>(tile, t, k);
                for (int b = 0; b < 3; ++b) {
                    double* o = sraw + ((int64_t)b * 5 + t) * nr + r;
                    if (wgt[b] != 0.0) *o += wgt[b] * st;
                    if (s == 0) *o *= scl;
                }
            }
        }
    }
}

template <typename T>
__global__ void __launch_bounds__(Pts<T>::THREADS)
    density_slice(const T* __restrict__ a, const T* __restrict__ c, DensityArgs d, int s, int want_s, ClassLists jl,
                  double* __restrict__ raw, double* __restrict__ junc, double* __restrict__ qend,
                  double* __restrict__ sraw) {
    density_slice_tiles<T>(a, c, d, s, want_s, jl, raw, junc, qend, sraw);
}

template <typename T>
__global__ void __launch_bounds__(Pts<T>::THREADS)
    density_slice_batched(const SliceBatchArgs<T>* __restrict__ args, int s) {
    const SliceBatchArgs<T> g = args[blockIdx.y];
    density_slice_tiles<T>(g.qf + (int64_t)s * g.sl, g.qb + (int64_t)(s & 3) * g.sl, g.d, s, g.want_s, g.jl, g.raw,
                           g.junc, g.qend, g.sraw);
}

// periodic Simpson weight product (utility_mod.f90:236-298): (h/3)*(2|4)
__device__ __forceinline__ double simpson_w(int64_t r, const S3Args& s) {
    const int x = (int)(r % s.n[0]);
    const int y = (int)((r / s.n[0]) % s.n[1]);
    const int z = (int)(r / ((int64_t)s.n[0] * s.n[1]));
    const double wx = (x & 1) ? 4.0 : 2.0, wy = (y & 1) ? 4.0 : 2.0, wz = (z & 1) ? 4.0 : 2.0;
    return (s.d[0] / 3.0 * wx) * (s.d[1] / 3.0 * wy) * (s.d[2] / 3.0 * wz);
}

// partial Simpson sums of sum_k a[k*stride + r] for k < nsum
__global__ void s3_partial(const double* __restrict__ a, int nsum, int64_t stride, S3Args s, double* __restrict__ part) {
    __shared__ double sh[256];
    const int64_t nr = (int64_t)s.n[0] * s.n[1] * s.n[2];
    const int64_t chunk = (nr + gridDim.x - 1) / gridDim.x;
    const int64_t beg = blockIdx.x * chunk, end = min(nr, beg + chunk);
    double acc = 0.0;
    for (int64_t r = beg + threadIdx.x; r < end; r += blockDim.x) {
        double v = 0.0;
        for (int k = 0; k < nsum; ++k) v += a[k * stride + r];
        acc += simpson_w(r, s) * v;
    }
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) part[blockIdx.x] = sh[0];
}

__global__ void sum_partials(const double* __restrict__ part, int n, double* __restrict__ out) {
    __shared__ double sh[256];
    double acc = 0.0;
    for (int k = threadIdx.x; k < n; k += blockDim.x) acc += part[k];
    sh[threadIdx.x] = acc;
    __syncthreads();
    for (int w = 128; w > 0; w >>= 1) {
        if (threadIdx.x < w) sh[threadIdx.x] += sh[threadIdx.x + w];
        __syncthreads();
    }
    if (threadIdx.x == 0) *out = sh[0];
}

__global__ void scale_by(double* __restrict__ a, int64_t n, const double* __restrict__ denom, double vol) {
    const double f = vol / *denom;
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        a[e] = a[e] * f;
}

// free-energy integrand, three-block form of SCFT_Density_FE.f90:296-320
__global__ void fe_integrand(const double* __restrict__ phi, const double* __restrict__ w,
                             const double* __restrict__ mop, FeArgs f, double* __restrict__ ar) {
    const int64_t nr = f.nr;
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nr; r += (int64_t)gridDim.x * blockDim.x) {
        const double pa = phi[r], pb = phi[nr + r], pc = phi[2 * nr + r];
        const double wa = w[r], wb = w[nr + r], wc = w[2 * nr + r];
        double v = f.chi[0] * pa * pb + f.chi[1] * pa * pc + f.chi[2] * pb * pc - wa * pa - wb * pb - wc * pc +
                   (wa + wb + wc) / 3.0 * (pa + pb + pc - 1.0);
        if (f.ms) {
            double dd = 0.0;
            for (int p = 0; p < 3; ++p)
                for (int q = 0; q < 3; ++q) dd += mop[(p * 3 + q) * nr + r] * mop[(q * 3 + p) * nr + r];
            v += 0.5 * (dd / f.nmu);
        }
        ar[r] = v;
    }
}

// One read and one write per value; expanding on the host took 40 ms of a
// 128^3 call (27 planes of 2 M points), the transfer itself 20 ms.
__global__ void s_planes(const double* __restrict__ s, double* __restrict__ out, int p0, int64_t nr) {
    const int p = p0 + blockIdx.y, b = p / 9, q = p % 9;
    const int8_t comp[9] = {0, 2, 3, 2, 1, 4, 3, 4, -1};
    const double* c = s + (int64_t)b * 5 * nr;
    double* o = out + (int64_t)blockIdx.y * nr;
    const int k = comp[q];
    for (int64_t r = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; r < nr; r += (int64_t)gridDim.x * blockDim.x)
        o[r] = k >= 0 ? c[k * nr + r] : -(c[r] + c[nr + r]);
}

__global__ void count_nonfinite(const double* __restrict__ a, int64_t n, int* __restrict__ flag) {
    for (int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; e < n; e += (int64_t)gridDim.x * blockDim.x)
        if (!isfinite(a[e])) atomicOr(flag, 1);
}

// ------------------------------------------------------------ launchers
static int grid_for(int64_t n) {
    int64_t g = (n + 255) / 256;
    return (int)(g > 4096 ? 4096 : (g < 1 ? 1 : g));
}

template <typename T> void launch_to_internal(const double* ref, T* out, int M, int64_t nr, cudaStream_t st) {
    dim3 g((unsigned)((nr + 31) / 32), (unsigned)((M + 31) / 32));
    to_internal<T><<<g, dim3(32, 8), 0, st>>>(ref, out, M, nr);
}
template <typename T> void launch_to_reference(const T* in, double* ref, int M, int64_t nr, cudaStream_t st) {
    dim3 g((unsigned)((nr + 31) / 32), (unsigned)((M + 31) / 32));
    to_reference<T><<<g, dim3(32, 8), 0, st>>>(in, ref, M, nr);
}
template <typename T> void launch_set_delta(T* q, int M, int64_t nr, cudaStream_t st) {
    set_delta<T><<<grid_for((int64_t)M * nr), 256, 0, st>>>(q, M, nr);
}
template <typename T> void launch_make_cf(const double* w, T* cf, double ds, double third, int64_t nr, cudaStream_t st) {
    make_cf<T><<<grid_for(nr), 256, 0, st>>>(w, cf, ds, third, nr);
}
// CTAs of the tiled kernels: enough to fill the GPU, each walking several
// tiles so that the staged lists are reused
static unsigned tile_grid(int64_t nr, int tile) {
    const int64_t tiles = (nr + tile - 1) / tile;
    return (unsigned)(tiles < 1216 ? (tiles < 1 ? 1 : tiles) : 1216);
}

template <typename T>
void launch_ms_term(const T* h1, const T* h2, const T* h3, int order, const double* mop, const ClassLists& tl,
                    double ds, double thresh, int M, int64_t nr, T* out, cudaStream_t st) {
    ms_term<T><<<tile_grid(nr, PointTile<T>::value), Pts<T>::THREADS, ms_smem_bytes<T>(tl, M), st>>>(
        h1, h2, h3, order, mop, tl, ds, thresh, M, nr, out);
}
template <typename T>
void launch_density(const T* qf, const T* qb, const DensityArgs& d, double* raw, double* junc, double* qend,
                    cudaStream_t st) {
    constexpr int P = Pts<T>::P;
    const int64_t nr = d.nr;
    // P points a thread once that makes 3 CTAs for every SM, with the coefficients
    // in two groups if need be; one point and eight groups on small grids
    if (nr / (256 * P) >= 456)
        density_accum<T, P, 1><<<(unsigned)((nr / P + 255) / 256), 256, 0, st>>>(qf, qb, d, raw, junc, qend);
    else if (nr / (128 * P) >= 456)
        density_accum<T, P, 2><<<(unsigned)((nr / P + 127) / 128), 256, 0, st>>>(qf, qb, d, raw, junc, qend);
    else
        density_accum<T, 1, 8><<<(unsigned)((nr + 31) / 32), 256, 0, st>>>(qf, qb, d, raw, junc, qend);
}
template <typename T>
void launch_stensor(const T* qf, const T* qb, const DensityArgs& d, const ClassLists& jl, double* sraw, cudaStream_t st) {
    stensor_accum<T><<<(unsigned)(d.nr / PointTile<T>::value), Pts<T>::THREADS, slice_smem_bytes<T>(jl, d.M, true), st>>>(
        qf, qb, d, jl, sraw);
}

template <typename T>
void launch_density_slice(const T* qf_s, const T* qb_s, const DensityArgs& d, int s, int want_s, const ClassLists& jl,
                          double* raw, double* junc, double* qend, double* sraw, cudaStream_t st) {
    density_slice<T><<<tile_grid(d.nr, PointTile<T>::value), Pts<T>::THREADS, slice_smem_bytes<T>(jl, d.M, want_s != 0),
                       st>>>(qf_s, qb_s, d, s, want_s, jl, raw, junc, qend, sraw);
}

template <typename T>
void launch_density_slice_batched(const SliceBatchArgs<T>* args, int count, int64_t max_nr, int s, int M,
                                  const ClassLists& jl, int any_s, cudaStream_t st) {
    density_slice_batched<T><<<dim3(tile_grid(max_nr, PointTile<T>::value), count), Pts<T>::THREADS,
                               slice_smem_bytes<T>(jl, M, any_s != 0), st>>>(args, s);
}

void launch_s3(const double* a, int nsum, int64_t stride, const S3Args& s, double* part, double* out,
               cudaStream_t st) {
    s3_partial<<<kS3Blocks, 256, 0, st>>>(a, nsum, stride, s, part);
    sum_partials<<<1, 256, 0, st>>>(part, kS3Blocks, out);
}

void launch_scale(double* a, int64_t n, const double* denom, double vol, cudaStream_t st) {
    scale_by<<<grid_for(n), 256, 0, st>>>(a, n, denom, vol);
}

void launch_fe(const double* phi, const double* w, const double* mop, const FeArgs& f, double* ar, cudaStream_t st) {
    fe_integrand<<<grid_for(f.nr), 256, 0, st>>>(phi, w, mop, f, ar);
}

void launch_s_planes(const double* s, double* out, int p0, int np, int64_t nr, cudaStream_t st) {
    s_planes<<<dim3(std::min(grid_for(nr), 512), np), 256, 0, st>>>(s, out, p0, nr);
}

void launch_nonfinite(const double* a, int64_t n, int* flag, cudaStream_t st) {
    count_nonfinite<<<grid_for(n), 256, 0, st>>>(a, n, flag);
}

#define WLC_INST(T)                                                                                              \
    template void launch_to_internal<T>(const double*, T*, int, int64_t, cudaStream_t);                           \
    template void launch_to_reference<T>(const T*, double*, int, int64_t, cudaStream_t);                          \
    template void launch_set_delta<T>(T*, int, int64_t, cudaStream_t);                                           \
    template void launch_make_cf<T>(const double*, T*, double, double, int64_t, cudaStream_t);                    \
    template void launch_ms_term<T>(const T*, const T*, const T*, int, const double*, const ClassLists&, double,  \
                                    double, int, int64_t, T*, cudaStream_t);                                     \
    template void launch_density<T>(const T*, const T*, const DensityArgs&, double*, double*, double*,           \
                                    cudaStream_t);                                                               \
    template void launch_stensor<T>(const T*, const T*, const DensityArgs&, const ClassLists&, double*, cudaStream_t); \
    template void launch_density_slice<T>(const T*, const T*, const DensityArgs&, int, int, const ClassLists&, double*, \
                                          double*, double*, double*, cudaStream_t);                              \
    template void launch_density_slice_batched<T>(const SliceBatchArgs<T>*, int, int64_t, int, int,                  \
                                                  const ClassLists&, int, cudaStream_t);
WLC_INST(double)
WLC_INST(float)
#undef WLC_INST

cudaError_t prepare_reduce_kernels() {
    // per (kernel, device): a context may be created on any device
    const int big = 200 * 1024;
    const void* fns[] = {(const void*)stensor_accum<double>, (const void*)stensor_accum<float>,
                         (const void*)density_slice<double>, (const void*)density_slice<float>,
                         (const void*)density_slice_batched<double>, (const void*)density_slice_batched<float>,
                         (const void*)ms_term<double>, (const void*)ms_term<float>};
    for (const void* fn : fns)
        if (const cudaError_t e = smem_attr_once(fn, big); e != cudaSuccess) return e;
    return cudaSuccess;
}

}  // namespace wlc
