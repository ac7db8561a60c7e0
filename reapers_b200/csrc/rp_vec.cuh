// Vector kernels (the BLAS-1 surface of the reference's Impl concept,
// inc/gpuimpl.h:853-1002) and the multi-vector kernels of block Gram-Schmidt.
#pragma once

#include "rp_common.cuh"

namespace rp {

constexpr int MAX_KRYLOV = 64;   // largest Krylov dimension (vectors u_0..u_m)

// Pointer table passed by value (kernel parameter space).
struct VecTable {
    const void *p[MAX_KRYLOV + 1];
};

// Vectors are streamed as 16-byte packets: one complex double or two complex
// floats.  A packet count of n * sizeof(element) / 16 leaves out the last element
// of an odd complex64 vector; k_dot adds it, the others take states, whose length
// is even.
template <typename Real>
struct Packet;
template <>
struct Packet<double> {
    static constexpr int E = 1;
    double2 v;
    __device__ __forceinline__ void load(const void *p, uint64_t k) {
        v = __ldg(static_cast<const double2 *>(p) + k);
    }
    __device__ __forceinline__ void load_rw(const void *p, uint64_t k) {
        v = static_cast<const double2 *>(p)[k];
    }
    __device__ __forceinline__ double re(int) const { return v.x; }
    __device__ __forceinline__ double im(int) const { return v.y; }
    __device__ __forceinline__ void set(int, double r, double i) { v = make_double2(r, i); }
    __device__ __forceinline__ void store(void *p, uint64_t k) const {
        static_cast<double2 *>(p)[k] = v;
    }
};
template <>
struct Packet<float> {
    static constexpr int E = 2;
    float4 v;
    __device__ __forceinline__ void load(const void *p, uint64_t k) {
        v = __ldg(static_cast<const float4 *>(p) + k);
    }
    __device__ __forceinline__ void load_rw(const void *p, uint64_t k) {
        v = static_cast<const float4 *>(p)[k];
    }
    __device__ __forceinline__ double re(int e) const { return e ? v.z : v.x; }
    __device__ __forceinline__ double im(int e) const { return e ? v.w : v.y; }
    __device__ __forceinline__ void set(int e, double r, double i) {
        if (e) {
            v.z = (float)r;
            v.w = (float)i;
        } else {
            v.x = (float)r;
            v.y = (float)i;
        }
    }
    __device__ __forceinline__ void store(void *p, uint64_t k) const {
        static_cast<float4 *>(p)[k] = v;
    }
};

#if defined(__CUDACC__)
// x += sum_{q < N} c_q u_q of packet k (c complex in shared memory).  The number
// of vectors is a template argument: a test on it in the loop let the compiler
// sink each load to its use, one in flight at a time (2.5x slower).
template <typename Real, int N>
__device__ __forceinline__ void axpy_group(double (&xr)[Packet<Real>::E], double (&xi)[Packet<Real>::E],
                                           const void *const *u, const double *c, uint64_t k) {
    Packet<Real> up[N];
#pragma unroll
    for (int q = 0; q < N; q++) up[q].load(u[q], k);
#pragma unroll
    for (int q = 0; q < N; q++) {
        const double cr = c[2 * q], ci = c[2 * q + 1];
#pragma unroll
        for (int e = 0; e < Packet<Real>::E; e++) {
            const double ur = up[q].re(e), ui = up[q].im(e);
            xr[e] = fma(cr, ur, fma(-ci, ui, xr[e]));
            xi[e] = fma(cr, ui, fma(ci, ur, xi[e]));
        }
    }
}

template <typename Real>
__device__ __forceinline__ void axpy_vectors(double (&xr)[Packet<Real>::E], double (&xi)[Packet<Real>::E],
                                             const void *const *u, const double *c, int n, uint64_t k) {
    for (; n >= 8; n -= 8, u += 8, c += 16) axpy_group<Real, 8>(xr, xi, u, c, k);
    switch (n) {
    case 7: axpy_group<Real, 7>(xr, xi, u, c, k); break;
    case 6: axpy_group<Real, 6>(xr, xi, u, c, k); break;
    case 5: axpy_group<Real, 5>(xr, xi, u, c, k); break;
    case 4: axpy_group<Real, 4>(xr, xi, u, c, k); break;
    case 3: axpy_group<Real, 3>(xr, xi, u, c, k); break;
    case 2: axpy_group<Real, 2>(xr, xi, u, c, k); break;
    case 1: axpy_group<Real, 1>(xr, xi, u, c, k); break;
    default: break;
    }
}
#endif

// Grid used by the reduction kernels; partial buffers hold grid * n * 2 doubles.
int reduce_grid();

void vec_convert(int dtype_dst, void *dst, int dtype_src, const void *src, uint64_t n,
                 cudaStream_t st);
void vec_axpy(int dtype, uint64_t n, void *y, double ar, double ai, const void *x,
              cudaStream_t st);
void vec_add3(int dtype, uint64_t n, void *res, const void *a, const void *b, cudaStream_t st);
void vec_scale(int dtype, uint64_t n, void *v, double ar, double ai, cudaStream_t st);
void vec_random(int dtype, uint64_t n, void *v, uint64_t seed, cudaStream_t st);

// out = <a|b> and sqrt(<v|v>) (FP64 sums, compensated over the CTAs), synchronous.
void vec_dot(int dtype, uint64_t n, const void *a, const void *b, double *out, cudaStream_t st);
double vec_norm(int dtype, uint64_t n, const void *v, cudaStream_t st);

// w += sum_i coef[i] * u_i (coef complex double on the device), i < nvec or
// i < *nvec_dev when nvec_dev is given; n even for complex64.
void multi_axpy(int dtype, uint64_t n, const VecTable &tab, int nvec, const int *nvec_dev,
                const double *coef, void *w, cudaStream_t st);

// Device scratch kept between calls: the step-size candidates' expm buffer, the
// dense matrix-vector product's column-chunk partials and the dense exponential's
// scaled eigenvectors.  A slot grows on demand (the stream is synchronised before a smaller buffer is
// freed); scratch_release_all(), called by rp_shutdown, frees every slot, so
// a later rp_init allocates them afresh.
enum ScratchSlot { SCR_EXPM = 0, SCR_MATVEC, SCR_EXPM_DENSE, SCR_COUNT };
void *scratch_get(int slot, size_t bytes, cudaStream_t st);
void scratch_release_all();

}  // namespace rp
