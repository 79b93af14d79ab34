// wlc_reduce.h -- launch interface of the layout, density and reduction
// kernels (wlc_reduce.cu).
#pragma once
#include <cstdint>
#include <cuda_runtime.h>

namespace wlc {

constexpr int kS3Blocks = 512;  // CTAs of the deterministic Simpson reduction

struct DensityArgs {
    int64_t nr;
    int M;
    int nmax;
    int nstart[3], ns[3];
    double ds;
};

struct S3Args {
    int n[3];
    double d[3];
};

struct FeArgs {
    int64_t nr;
    double chi[3];  // AB, AC, BC
    double nmu;
    int ms;
};

// Sparse coupling tensors of five components, row by row and component by
// component: entries of (row i, component c) at [ptr[5i+c], ptr[5i+c+1]).
// Theta: components T1122, T33, T12, T13, T23; pairs (i, j) with several
// nonzero components are kept apart (g*, all five values), because the
// threshold applies to their sum.  J: components (J11+J22)/2, (J11-J22)/2,
// J12, J13, J23 (for one pair (i, j) most components vanish: m of the two
// harmonics picks one).
struct ClassLists {
    int n, ng;
    const uint16_t* ptr;    // [5M + 1]
    const int16_t* col;
    const double* val;
    double vmin[5], vmax[5];  // |val| over each component
    const uint16_t* gptr;   // [M + 1]
    const int16_t* gcol;
    const double* gval;     // [ng][5]
    const int16_t* order;   // rows, longest first
};

// points per CTA of the tiled per-point coefficient kernels (ms_term,
// density slices, orientation tensor): the coefficient vectors of the tile
// are staged in shared memory once
template <typename T> struct PointTile {
    static constexpr int value = sizeof(T) == 8 ? 32 : 64;
};
// function attributes of the tiled kernels (large shared memory) on the
// current device; call on each device before any stream capture (repeat
// calls on a device return at once)
cudaError_t prepare_reduce_kernels();

template <typename T> void launch_to_internal(const double* ref, T* out, int M, int64_t nr, cudaStream_t st);
template <typename T> void launch_to_reference(const T* in, double* ref, int M, int64_t nr, cudaStream_t st);
template <typename T> void launch_set_delta(T* q, int M, int64_t nr, cudaStream_t st);
template <typename T>
void launch_make_cf(const double* w, T* cf, double ds, double third, int64_t nr, cudaStream_t st);
template <typename T>
void launch_ms_term(const T* h1, const T* h2, const T* h3, int order, const double* mop, const ClassLists& tl,
                    double ds, double thresh, int M, int64_t nr, T* out, cudaStream_t st);
template <typename T>
void launch_density(const T* qf, const T* qb, const DensityArgs& d, double* raw, double* junc, double* qend,
                    cudaStream_t st);
template <typename T>
void launch_stensor(const T* qf, const T* qb, const DensityArgs& d, const ClassLists& jl, double* sraw, cudaStream_t st);
// one contour slice s of the streamed density integrals (q(s), q*(s) given):
// raw/sraw += Simpson weight x q.q* for the blocks containing s, junction
// and Q(end) slices copied; at the last slice (s = 0) scaled by ds/3
// per-instance arguments of a batched density_slice launch (instance j =
// blockIdx.y): q(s) = qf + s*sl, q*(s) = qb + (s & 3)*sl (streamed ring)
template <typename T> struct SliceBatchArgs {
    const T* qf;
    const T* qb;
    int64_t sl;
    DensityArgs d;
    int want_s;
    ClassLists jl;
    double* raw;
    double* junc;
    double* qend;
    double* sraw;
};
template <typename T>
void launch_density_slice_batched(const SliceBatchArgs<T>* args, int count, int64_t max_nr, int s, int M,
                                  const ClassLists& jl, int any_s, cudaStream_t st);

template <typename T>
void launch_density_slice(const T* qf_s, const T* qb_s, const DensityArgs& d, int s, int want_s, const ClassLists& jl,
                          double* raw, double* junc, double* qend, double* sraw, cudaStream_t st);
void launch_s3(const double* a, int nsum, int64_t stride, const S3Args& s, double* part, double* out,
               cudaStream_t st);
void launch_scale(double* a, int64_t n, const double* denom, double vol, cudaStream_t st);
void launch_fe(const double* phi, const double* w, const double* mop, const FeArgs& f, double* ar, cudaStream_t st);
// planes p0 .. p0+np-1 of S_OP(r, a, b, blk) (plane a + 3b + 9 blk) from the
// components s[blk][5][nr] (xx, yy, xy, xz, yz); S_zz = -(S_xx + S_yy)
void launch_s_planes(const double* s, double* out, int p0, int np, int64_t nr, cudaStream_t st);
void launch_nonfinite(const double* a, int64_t n, int* flag, cudaStream_t st);

}  // namespace wlc
