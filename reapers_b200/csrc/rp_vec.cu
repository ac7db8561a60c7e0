// Vector kernels: conversion, axpy, scaling, random states, inner products and
// linear combinations of basis vectors.
// All reductions accumulate in FP64 (products of FP32 operands are exact in
// FP64) with a compensated fixed-order combination across warps and CTAs, so
// results are reproducible run to run.
#include <cmath>

#include "rp_apply.cuh"
#include "rp_vec.cuh"

namespace rp {

int reduce_grid() { return 2 * num_sms(); }

static void *g_scratch[SCR_COUNT] = {};
static size_t g_scratch_cap[SCR_COUNT] = {};

void *scratch_get(int slot, size_t bytes, cudaStream_t st) {
    if (bytes > g_scratch_cap[slot]) {
        if (g_scratch[slot]) {
            RP_CUDA(cudaStreamSynchronize(st));
            cudaFree(g_scratch[slot]);
        }
        g_scratch[slot] = nullptr;
        g_scratch_cap[slot] = 0;
        RP_CUDA(cudaMalloc(&g_scratch[slot], bytes));
        g_scratch_cap[slot] = bytes;
    }
    return g_scratch[slot];
}

static void dot_scratch_release();

void scratch_release_all() {
    dot_scratch_release();
    for (int s = 0; s < SCR_COUNT; s++) {
        if (g_scratch[s]) cudaFree(g_scratch[s]);
        g_scratch[s] = nullptr;
        g_scratch_cap[s] = 0;
    }
}

static inline int blocks_for(uint64_t n, int threads, int cap) {
    uint64_t b = (n + threads - 1) / threads;
    return (int)(b < (uint64_t)cap ? (b ? b : 1) : cap);
}

template <typename RO, typename RI>
__global__ void k_convert(Cplx<RO> *dst, const Cplx<RI> *src, uint64_t n) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        Cplx<RI> v = src[i];
        dst[i] = Cplx<RO>{(RO)v.x, (RO)v.y};   // round to nearest
    }
}

void vec_convert(int dto, void *dst, int dfrom, const void *src, uint64_t n, cudaStream_t st) {
    if (!n) return;
    const int bl = blocks_for(n, 256, 8 * num_sms());
    if (dto == dfrom) {
        RP_CUDA(cudaMemcpyAsync(dst, src, n * (dto == 2 ? 16 : 8), cudaMemcpyDeviceToDevice, st));
    } else if (dto == 1) {
        k_convert<float, double><<<bl, 256, 0, st>>>((Cplx<float> *)dst, (const Cplx<double> *)src, n);
    } else {
        k_convert<double, float><<<bl, 256, 0, st>>>((Cplx<double> *)dst, (const Cplx<float> *)src, n);
    }
    RP_CUDA(cudaGetLastError());
}

template <typename Real>
__global__ void k_axpy(uint64_t n, Cplx<Real> *y, double ar, double ai, const Cplx<Real> *x) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        Cplx<Real> v = x[i], w = y[i];
        w.x = (Real)((double)w.x + ar * v.x - ai * v.y);
        w.y = (Real)((double)w.y + ar * v.y + ai * v.x);
        y[i] = w;
    }
}

void vec_axpy(int dtype, uint64_t n, void *y, double ar, double ai, const void *x,
              cudaStream_t st) {
    if (!n) return;
    const int bl = blocks_for(n, 256, 8 * num_sms());
    if (dtype == 2) k_axpy<double><<<bl, 256, 0, st>>>(n, (Cplx<double> *)y, ar, ai, (const Cplx<double> *)x);
    else k_axpy<float><<<bl, 256, 0, st>>>(n, (Cplx<float> *)y, ar, ai, (const Cplx<float> *)x);
    RP_CUDA(cudaGetLastError());
}

template <typename Real>
__global__ void k_add3(uint64_t n, Cplx<Real> *r, const Cplx<Real> *a, const Cplx<Real> *b) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        Cplx<Real> u = a[i], v = b[i];
        r[i] = Cplx<Real>{u.x + v.x, u.y + v.y};
    }
}

void vec_add3(int dtype, uint64_t n, void *res, const void *a, const void *b, cudaStream_t st) {
    if (!n) return;
    const int bl = blocks_for(n, 256, 8 * num_sms());
    if (dtype == 2) k_add3<double><<<bl, 256, 0, st>>>(n, (Cplx<double> *)res, (const Cplx<double> *)a, (const Cplx<double> *)b);
    else k_add3<float><<<bl, 256, 0, st>>>(n, (Cplx<float> *)res, (const Cplx<float> *)a, (const Cplx<float> *)b);
    RP_CUDA(cudaGetLastError());
}

template <typename Real>
__global__ void k_scale(uint64_t n, Cplx<Real> *v, double ar, double ai) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        Cplx<Real> w = v[i];
        v[i] = Cplx<Real>{(Real)(ar * w.x - ai * w.y), (Real)(ar * w.y + ai * w.x)};
    }
}

void vec_scale(int dtype, uint64_t n, void *v, double ar, double ai, cudaStream_t st) {
    if (!n) return;
    const int bl = blocks_for(n, 256, 8 * num_sms());
    if (dtype == 2) k_scale<double><<<bl, 256, 0, st>>>(n, (Cplx<double> *)v, ar, ai);
    else k_scale<float><<<bl, 256, 0, st>>>(n, (Cplx<float> *)v, ar, ai);
    RP_CUDA(cudaGetLastError());
}

// Counter-based normal deviates: splitmix64 hash of (seed, index) -> two
// uniforms -> Box-Muller.  Deterministic for a given seed.
__device__ __forceinline__ uint64_t splitmix64(uint64_t x) {
    x += 0x9E3779B97F4A7C15ull;
    x = (x ^ (x >> 30)) * 0xBF58476D1CE4E5B9ull;
    x = (x ^ (x >> 27)) * 0x94D049BB133111EBull;
    return x ^ (x >> 31);
}

template <typename Real>
__global__ void k_random(uint64_t n, Cplx<Real> *v, uint64_t seed) {
    for (uint64_t i = blockIdx.x * (uint64_t)blockDim.x + threadIdx.x; i < n;
         i += (uint64_t)gridDim.x * blockDim.x) {
        uint64_t h1 = splitmix64(seed * 0x632BE59BD9B4E019ull + 2 * i);
        uint64_t h2 = splitmix64(seed * 0x632BE59BD9B4E019ull + 2 * i + 1);
        double u1 = ((h1 >> 11) + 1) * (1.0 / 9007199254740993.0);   // (0, 1]
        double u2 = (h2 >> 11) * (1.0 / 9007199254740992.0);         // [0, 1)
        double r = sqrt(-2.0 * log(u1));
        double s, c;
        sincospi(2.0 * u2, &s, &c);
        v[i] = Cplx<Real>{(Real)(r * c), (Real)(r * s)};
    }
}

void vec_random(int dtype, uint64_t n, void *v, uint64_t seed, cudaStream_t st) {
    if (!n) return;
    const int bl = blocks_for(n, 256, 8 * num_sms());
    if (dtype == 2) k_random<double><<<bl, 256, 0, st>>>(n, (Cplx<double> *)v, seed);
    else k_random<float><<<bl, 256, 0, st>>>(n, (Cplx<float> *)v, seed);
    RP_CUDA(cudaGetLastError());
}

// ---------------------------------------------------------------------------
// Inner product and linear combination
// ---------------------------------------------------------------------------
constexpr int RT = 256;   // threads of the reduction kernels
constexpr int RW = RT / 32;

// <a|b> (a norm is <v|v>, its second load of a packet served by L1): a CTA sums
// every gridDim-th stretch of packets, four loads of each vector in flight per
// thread; the last CTA to arrive adds the CTAs' partials
// (compensated, fixed order) and writes the pair to pinned host memory, so a
// call is one launch and one synchronisation.  (Two kernels, the second adding
// 296 partials in one thread, and a copy: 30 us on the device for 2^16
// elements; now 5.)
template <typename Real>
__global__ void __launch_bounds__(RT) k_dot(uint64_t n, const void *a, const void *b, double *partials,
                                            unsigned *arrived, double *out) {
    constexpr int E = Packet<Real>::E, U = 4;
    __shared__ double scratch[RW][2];
    __shared__ bool s_last;
    const uint64_t npk = n / E, stride = (uint64_t)gridDim.x * RT;
    double sr = 0.0, si = 0.0;
    auto add = [&](double ar, double ai, double br, double bi) {
        sr = fma(ar, br, fma(ai, bi, sr));
        si = fma(ar, bi, fma(-ai, br, si));
    };
    uint64_t k = blockIdx.x * (uint64_t)RT + threadIdx.x;
    for (; k + (U - 1) * stride < npk; k += U * stride) {
        Packet<Real> x[U], y[U];
#pragma unroll
        for (int u = 0; u < U; u++) {
            x[u].load(a, k + u * stride);
            y[u].load(b, k + u * stride);
        }
#pragma unroll
        for (int u = 0; u < U; u++) {
#pragma unroll
            for (int e = 0; e < E; e++) add(x[u].re(e), x[u].im(e), y[u].re(e), y[u].im(e));
        }
    }
    for (; k < npk; k += stride) {
        Packet<Real> x, y;
        x.load(a, k);
        y.load(b, k);
#pragma unroll
        for (int e = 0; e < E; e++) add(x.re(e), x.im(e), y.re(e), y.im(e));
    }
    if (n % E && blockIdx.x == 0 && threadIdx.x == 0) {   // the odd complex64 element
        const Cplx<Real> x = static_cast<const Cplx<Real> *>(a)[n - 1];
        const Cplx<Real> y = static_cast<const Cplx<Real> *>(b)[n - 1];
        add(x.x, x.y, y.x, y.y);
    }
    sr = warp_sum(sr);
    si = warp_sum(si);
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (lane == 0) {
        scratch[warp][0] = sr;
        scratch[warp][1] = si;
    }
    __syncthreads();
    if (threadIdx.x < 2) {
        CompSum c;
        for (int w = 0; w < RW; w++) c.add(scratch[w][threadIdx.x]);
        partials[2 * blockIdx.x + threadIdx.x] = c.value();
        __threadfence();
    }
    __syncthreads();
    // atomicInc wraps to 0 with the last arrival: ready for the next launch
    if (threadIdx.x == 0) s_last = atomicInc(arrived, gridDim.x - 1) == gridDim.x - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (warp < 2) {
        const double v = warp_compsum(partials + warp, gridDim.x, 2);
        if (lane == 0) out[warp] = v;
    }
}

// Partials, arrival count (device) and result (pinned host) of vec_dot; the
// calls run one after the other (the library's lock and stream).
struct DotScratch {
    double *partials = nullptr;
    unsigned *arrived = nullptr;
    double *out = nullptr;
};
static DotScratch g_dot;

static void dot_scratch_release() {
    if (g_dot.partials) cudaFree(g_dot.partials);
    if (g_dot.out) cudaFreeHost(g_dot.out);
    g_dot = DotScratch{};
}

void vec_dot(int dtype, uint64_t n, const void *a, const void *b, double *out, cudaStream_t st) {
    if (!g_dot.out) {
        const size_t pb = (size_t)reduce_grid() * 2 * sizeof(double);
        RP_CUDA(cudaMalloc((void **)&g_dot.partials, pb + sizeof(unsigned)));
        g_dot.arrived = reinterpret_cast<unsigned *>(reinterpret_cast<char *>(g_dot.partials) + pb);
        RP_CUDA(cudaMemset(g_dot.arrived, 0, sizeof(unsigned)));
        RP_CUDA(cudaHostAlloc((void **)&g_dot.out, 2 * sizeof(double), cudaHostAllocMapped));
    }
    // a CTA per 1024 packets while there are few, two per SM at most
    const int g = blocks_for(dtype == 2 ? n : n / 2, 4 * RT, reduce_grid());
    if (dtype == 2) k_dot<double><<<g, RT, 0, st>>>(n, a, b, g_dot.partials, g_dot.arrived, g_dot.out);
    else k_dot<float><<<g, RT, 0, st>>>(n, a, b, g_dot.partials, g_dot.arrived, g_dot.out);
    RP_CUDA(cudaGetLastError());
    RP_CUDA(cudaStreamSynchronize(st));
    out[0] = g_dot.out[0];
    out[1] = g_dot.out[1];
}

double vec_norm(int dtype, uint64_t n, const void *v, cudaStream_t st) {
    double out[2];
    vec_dot(dtype, n, v, v, out, st);
    return std::sqrt(out[0]);
}

// w += sum_i c_i u_i in one pass: per packet of w, the vectors are read in
// groups of eight independent 16-byte loads (axpy_vectors), the update is
// accumulated in FP64 and rounded once to the vector precision.
template <typename Real>
__global__ void __launch_bounds__(RT) k_multi_axpy(uint64_t npk, const VecTable tab, int nvec,
                                                   const int *nvec_dev, const double *coef, void *w) {
    constexpr int E = Packet<Real>::E;
    __shared__ double c[2 * (MAX_KRYLOV + 1)];
    const int nv = nvec_dev ? *nvec_dev : nvec;
    for (int i = threadIdx.x; i < 2 * nv; i += RT) c[i] = coef[i];
    __syncthreads();
    const uint64_t chunk = (npk + gridDim.x - 1) / gridDim.x;
    const uint64_t lo = blockIdx.x * chunk;
    const uint64_t hi = lo + chunk < npk ? lo + chunk : npk;
    for (uint64_t k = lo + threadIdx.x; k < hi; k += RT) {
        Packet<Real> wp;
        wp.load_rw(w, k);
        double xr[E], xi[E];
#pragma unroll
        for (int e = 0; e < E; e++) {
            xr[e] = wp.re(e);
            xi[e] = wp.im(e);
        }
        axpy_vectors<Real>(xr, xi, tab.p, c, nv, k);
#pragma unroll
        for (int e = 0; e < E; e++) wp.set(e, xr[e], xi[e]);
        wp.store(w, k);
    }
}

void multi_axpy(int dtype, uint64_t n, const VecTable &tab, int nvec, const int *nvec_dev,
                const double *coef, void *w, cudaStream_t st) {
    RP_REQUIRE(nvec >= 0 && nvec <= MAX_KRYLOV + 1, -2, "too many vectors");
    // six CTAs of 40 registers per SM (two per SM, as many as the reductions
    // take: 1.4x slower)
    const int g = blocks_for(dtype == 2 ? n : n / 2, RT, 6 * num_sms());
    if (dtype == 2)
        k_multi_axpy<double><<<g, RT, 0, st>>>(n, tab, nvec, nvec_dev, coef, w);
    else   // states have 2^len elements, len >= 1
        k_multi_axpy<float><<<g, RT, 0, st>>>(n / 2, tab, nvec, nvec_dev, coef, w);
    RP_CUDA(cudaGetLastError());
}

}  // namespace rp
