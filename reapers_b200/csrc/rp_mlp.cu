// Small MLP (in -> 64 -> 64 -> out, tanh hidden layers, linear output) for
// the learned Krylov step controller: hand-written CUDA forward, backward and
// Adam, FP32.  Parameters are one flat array
// [W1 (64 x in), b1, W2 (64 x 64), b2, W3 (out x 64), b3], row-major.
//
// An epoch of training is one cooperative launch (of up to 2^16 steps).  Per
// mini-batch every CTA takes the parameters into shared memory, runs its samples
// forward and backward four at a time (thread = hidden unit x sample) and writes its
// gradient partial, products and sums over samples in FP64; after a grid barrier
// the CTAs share the parameters out, sum the partials in a fixed order and apply
// Adam (reproducible); after another the next batch starts.  Loss: mean squared
// error / 2.
//
// A batch of 512 is 17 MFLOP: bound by latency (two barriers, the dependent
// layers), so the design counts launches, host round trips and bank conflicts:
// weight rows are padded to an odd length in shared memory, the samples stay on
// the device, an epoch uploads its order alone, and what the FP64 gradient
// multiplies is converted once per sweep.  Measured, 21 inputs, us per batch of
// 64 / 512 / 2048 / 8192, three kernels and a host sync per batch -> this: 47.7 /
// 86.3 / 199 / 458 -> 13.7 / 16.7 / 37.9 / 71.2 (with FP32 sums over a CTA's samples
// 13.2 / 17.3 / 34.8 / 64.9, and a gradient further from 64 bits than the former).
#include <cmath>
#include <vector>

#include "rp_apply.cuh"
#include "rp_common.cuh"
#include "rp_mlp.cuh"

namespace rp {

constexpr int HID = MLP_HIDDEN;

int mlp_num_params(int in, int out) { return HID * in + HID + HID * HID + HID + out * HID + out; }

struct MlpDims {
    int in, out, np;
    int oW1, ob1, oW2, ob2, oW3, ob3;
};

static MlpDims dims(int in, int out) {
    MlpDims d;
    d.in = in;
    d.out = out;
    d.oW1 = 0;
    d.ob1 = d.oW1 + HID * in;
    d.oW2 = d.ob1 + HID;
    d.ob2 = d.oW2 + HID * HID;
    d.oW3 = d.ob2 + HID;
    d.ob3 = d.oW3 + out * HID;
    d.np = d.ob3 + out;
    return d;
}

constexpr int MT = 256;                  // threads per CTA: 64 hidden units x MS samples
constexpr int MS = MT / HID;
constexpr int LD2 = HID + 1;             // row of W2 in shared memory

// Shared-memory image of the network and the activations of MS samples.
struct MlpShared {
    float *w1, *b1, *w2, *b2, *w3, *b3;  // w1 rows of in | 1, w2 rows of LD2
    float *x, *h1, *h2, *y, *dy, *dh2, *dh1;
    int ld1;
};

__host__ __device__ inline size_t mlp_shared_floats(const MlpDims &d) {
    return (size_t)HID * (d.in | 1) + HID + HID * LD2 + HID + d.out * HID + 8 +
           (size_t)MS * ((d.in + 3) & ~3) + 4 * MS * HID + 2 * MS * 8;
}

__device__ __forceinline__ MlpShared mlp_carve(const MlpDims &d, float *p) {
    MlpShared s;
    s.ld1 = d.in | 1;
    s.w1 = p, p += HID * s.ld1;
    s.b1 = p, p += HID;
    s.w2 = p, p += HID * LD2;
    s.b2 = p, p += HID;
    s.w3 = p, p += d.out * HID;
    s.b3 = p, p += 8;
    s.x = p, p += MS * ((d.in + 3) & ~3);
    s.h1 = p, p += MS * HID;
    s.h2 = p, p += MS * HID;
    s.dh2 = p, p += MS * HID;
    s.dh1 = p, p += MS * HID;
    s.y = p, p += MS * 8;
    s.dy = p;
    return s;
}

// The training kernel's FP64 copies of what the gradient multiplies (a value is
// converted once per sweep, not once per product), and, when it fits, the
// gradient itself.
struct MlpShared64 {
    double *x, *h1, *h2, *dy, *dh2, *dh1, *g;
};

__host__ __device__ inline size_t mlp_shared_at64(const MlpDims &d) {
    return (mlp_shared_floats(d) * sizeof(float) + 7) & ~(size_t)7;
}
__host__ __device__ inline size_t mlp_shared_doubles(const MlpDims &d) {
    return (size_t)MS * ((d.in + 3) & ~3) + 4 * MS * HID + MS * 8;
}

__device__ __forceinline__ MlpShared64 mlp_carve64(const MlpDims &d, void *sm) {
    double *p = reinterpret_cast<double *>(static_cast<char *>(sm) + mlp_shared_at64(d));
    MlpShared64 s;
    s.x = p, p += MS * ((d.in + 3) & ~3);
    s.h1 = p, p += MS * HID;
    s.h2 = p, p += MS * HID;
    s.dh2 = p, p += MS * HID;
    s.dh1 = p, p += MS * HID;
    s.dy = p, p += MS * 8;
    s.g = p;
    return s;
}

// The parameters, which other CTAs may just have written, from L2.
__device__ __forceinline__ void mlp_params(const MlpDims &d, const float *P, const MlpShared &s) {
    for (int i = threadIdx.x; i < HID * d.in; i += MT) s.w1[(i / d.in) * s.ld1 + i % d.in] = __ldcg(P + d.oW1 + i);
    for (int i = threadIdx.x; i < HID * HID; i += MT) s.w2[(i / HID) * LD2 + i % HID] = __ldcg(P + d.oW2 + i);
    for (int i = threadIdx.x; i < HID; i += MT) {
        s.b1[i] = __ldcg(P + d.ob1 + i);
        s.b2[i] = __ldcg(P + d.ob2 + i);
    }
    for (int i = threadIdx.x; i < d.out * HID; i += MT) s.w3[i] = __ldcg(P + d.oW3 + i);
    for (int i = threadIdx.x; i < d.out; i += MT) s.b3[i] = __ldcg(P + d.ob3 + i);
}

// Rows [at, at + ns) of X (through the order idx when given) into s.x.
__device__ __forceinline__ void mlp_rows(const MlpDims &d, const float *X, const int *idx, int at, int ns,
                                         const MlpShared &s) {
    const int ldx = (d.in + 3) & ~3;
    for (int i = threadIdx.x; i < MS * d.in; i += MT) {
        const int k = i / d.in, c = i % d.in;
        const int row = k < ns ? (idx ? idx[at + k] : at + k) : -1;
        s.x[k * ldx + c] = row >= 0 ? X[(size_t)row * d.in + c] : 0.f;
    }
}

// Forward for the MS samples in s.x: thread (k, j) = sample k, hidden unit j.
__device__ __forceinline__ void mlp_fwd(const MlpDims &d, const MlpShared &s) {
    const int j = threadIdx.x & (HID - 1), k = threadIdx.x / HID;
    const int ldx = (d.in + 3) & ~3;
    float a = s.b1[j];
    for (int i = 0; i < d.in; i++) a = fmaf(s.w1[j * s.ld1 + i], s.x[k * ldx + i], a);
    s.h1[k * HID + j] = tanhf(a);
    __syncthreads();
    float b = s.b2[j];
#pragma unroll 16
    for (int i = 0; i < HID; i++) b = fmaf(s.w2[j * LD2 + i], s.h1[k * HID + i], b);
    s.h2[k * HID + j] = tanhf(b);
    __syncthreads();
    if (threadIdx.x < MS * d.out) {
        const int kk = threadIdx.x / d.out, o = threadIdx.x % d.out;
        float c = s.b3[o];
#pragma unroll 16
        for (int i = 0; i < HID; i++) c = fmaf(s.w3[o * HID + i], s.h2[kk * HID + i], c);
        s.y[kk * 8 + o] = c;
    }
    __syncthreads();
}

__global__ void __launch_bounds__(MT) k_mlp_forward(MlpDims d, const float *params, const float *X,
                                                    int n, float *Y) {
    extern __shared__ float sm[];
    const MlpShared s = mlp_carve(d, sm);
    mlp_params(d, params, s);
    for (int at = blockIdx.x * MS; at < n; at += gridDim.x * MS) {
        const int ns = min(MS, n - at);
        __syncthreads();
        mlp_rows(d, X, nullptr, at, ns, s);
        __syncthreads();
        mlp_fwd(d, s);
        for (int i = threadIdx.x; i < ns * d.out; i += MT)
            Y[(size_t)at * d.out + i] = s.y[(i / d.out) * 8 + i % d.out];
    }
}

struct MlpSteps {
    const float *X, *Y;
    const int *idx;                      // order of the samples (null: as they lie)
    int n, batch;
    int parts;                           // CTAs that take samples; the others only update
    float *params, *m, *v, *g;
    int update;                          // 0: the gradient alone, into g
    float lr;
    int step0;                           // Adam steps taken before
    double *gpart, *lpart;               // [cta][np], [cta]
    float *loss;                         // [batch]
    int g_shared;                        // the gradient of several sweeps fits in shared memory
    unsigned *barrier, *err;
};

__global__ void __launch_bounds__(MT) k_mlp_steps(MlpDims d, const MlpSteps a) {
    extern __shared__ float sm[];
    const MlpShared s = mlp_carve(d, sm);
    const MlpShared64 v = mlp_carve64(d, sm);
    __shared__ double red[MS][HID];
    const int tid = threadIdx.x, j = tid & (HID - 1), k = tid / HID;
    const int ldx = (d.in + 3) & ~3;
    const int nsteps = (a.n + a.batch - 1) / a.batch;
    for (int step = 0; step < nsteps; step++) {
        const int b0 = step * a.batch, nb = min(a.batch, a.n - b0);
        const int per = (nb + a.parts - 1) / a.parts;
        const int nparts = (nb + per - 1) / per;
        if ((int)blockIdx.x < nparts) {
            const int s0 = b0 + (int)blockIdx.x * per, s1 = min(b0 + nb, s0 + per);
            // this CTA's partial, written as it is summed if one sweep makes it
            double *const part = a.gpart + (size_t)blockIdx.x * d.np;
            double *const G = a.g_shared && s1 - s0 > MS ? v.g : part;
            mlp_params(d, a.params, s);
            double loss = 0.0;
            for (int at = s0; at < s1; at += MS) {
                const int ns = min(MS, s1 - at);
                __syncthreads();
                mlp_rows(d, a.X, a.idx, at, ns, s);
                __syncthreads();
                mlp_fwd(d, s);
                if (tid < MS * 8) {
                    const int kk = tid >> 3, o = tid & 7;
                    float e = 0.f;
                    if (kk < ns && o < d.out) {
                        const int row = a.idx ? a.idx[at + kk] : at + kk;
                        e = s.y[kk * 8 + o] - a.Y[(size_t)row * d.out + o];
                        loss += (double)(0.5f * e * e);
                    }
                    s.dy[tid] = e;
                    v.dy[tid] = e;
                }
                for (int i = tid; i < MS * ldx; i += MT) v.x[i] = s.x[i];
                v.h1[tid] = s.h1[tid];
                v.h2[tid] = s.h2[tid];
                __syncthreads();
                float g2 = 0.f;
                for (int o = 0; o < d.out; o++) g2 = fmaf(s.w3[o * HID + j], s.dy[k * 8 + o], g2);
                const float h2 = s.h2[k * HID + j];
                const float dh2 = g2 * (1.f - h2 * h2);
                s.dh2[k * HID + j] = dh2;
                v.dh2[k * HID + j] = dh2;
                __syncthreads();
                float g1 = 0.f;
#pragma unroll 16
                for (int i = 0; i < HID; i++) g1 = fmaf(s.w2[i * LD2 + j], s.dh2[k * HID + i], g1);
                const float h1 = s.h1[k * HID + j];
                v.dh1[k * HID + j] = g1 * (1.f - h1 * h1);
                __syncthreads();
                // gradient entries, each one thread's own: products and sums in FP64
                const bool more = at > s0;
                double hq[MS];
#pragma unroll
                for (int q = 0; q < MS; q++) hq[q] = v.h1[q * HID + j];
#pragma unroll 4
                for (int r = k; r < HID; r += MS) {
                    double *const g = G + d.oW2 + r * HID + j;
                    double t = more ? *g : 0.0;
#pragma unroll
                    for (int q = 0; q < MS; q++) t = fma(v.dh2[q * HID + r], hq[q], t);
                    *g = t;
                }
                for (int i = tid; i < HID * d.in; i += MT) {
                    const int r = i / d.in, c = i - r * d.in;
                    double t = more ? G[d.oW1 + i] : 0.0;
#pragma unroll
                    for (int q = 0; q < MS; q++) t = fma(v.dh1[q * HID + r], v.x[q * ldx + c], t);
                    G[d.oW1 + i] = t;
                }
                for (int i = tid; i < d.out * HID; i += MT) {
                    double t = more ? G[d.oW3 + i] : 0.0;
#pragma unroll
                    for (int q = 0; q < MS; q++) t = fma(v.dy[q * 8 + i / HID], v.h2[q * HID + i % HID], t);
                    G[d.oW3 + i] = t;
                }
                if (tid < HID) {
                    double t1 = more ? G[d.ob1 + tid] : 0.0, t2 = more ? G[d.ob2 + tid] : 0.0;
#pragma unroll
                    for (int q = 0; q < MS; q++) t1 += v.dh1[q * HID + tid], t2 += v.dh2[q * HID + tid];
                    G[d.ob1 + tid] = t1;
                    G[d.ob2 + tid] = t2;
                }
                if (tid < d.out) {
                    double t = more ? G[d.ob3 + tid] : 0.0;
#pragma unroll
                    for (int q = 0; q < MS; q++) t += v.dy[q * 8 + tid];
                    G[d.ob3 + tid] = t;
                }
            }
            if (G != part) {
                __syncthreads();
                for (int i = tid; i < d.np; i += MT) part[i] = G[i];
            }
            if (tid < 32) {              // MS * 8 = 32 threads hold the loss
                loss = warp_sum(loss);
                if (tid == 0) a.lpart[blockIdx.x] = loss;
            }
        }
        if (!grid_barrier(a.barrier, a.err)) return;
        // this CTA's parameters: HID at a time, MS threads to a parameter
        const int share = (d.np + (int)gridDim.x - 1) / (int)gridDim.x;
        const int p0 = (int)blockIdx.x * share, p1 = min(d.np, p0 + share);
        const float c1 = 1.f - powf(0.9f, (float)(a.step0 + step + 1));
        const float c2 = 1.f - powf(0.999f, (float)(a.step0 + step + 1));
        for (int base = p0; base < p1; base += HID) {
            const int i = base + j;
            double sum = 0.0;
            if (i < p1) {
#pragma unroll 8
                for (int p = k; p < nparts; p += MS) sum += __ldcg(a.gpart + (size_t)p * d.np + i);
            }
            red[k][j] = sum;
            __syncthreads();
            if (k == 0 && i < p1) {
                double t = 0.0;
                for (int q = 0; q < MS; q++) t += red[q][j];
                const float g = (float)(t * (double)(1.f / nb));
                if (a.update) {
                    const float mi = 0.9f * a.m[i] + (1.f - 0.9f) * g;
                    const float vi = 0.999f * a.v[i] + (1.f - 0.999f) * g * g;
                    a.m[i] = mi;
                    a.v[i] = vi;
                    a.params[i] -= a.lr * (mi / c1) / (sqrtf(vi / c2) + 1e-8f);
                } else {
                    a.g[i] = g;
                }
            }
            __syncthreads();
        }
        if (blockIdx.x == 0 && tid < 32) {
            const double l = warp_compsum(a.lpart, nparts, 1);
            if (tid == 0) a.loss[step] = (float)(l / nb);
        }
        if (step + 1 < nsteps && !grid_barrier(a.barrier, a.err)) return;
    }
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------
static size_t fwd_smem(const MlpDims &d) { return mlp_shared_floats(d) * sizeof(float); }
// Training: the FP64 copies, and the gradient of a batch that takes several sweeps
// if it fits beside them (up to 190 inputs; else it is summed in its partial, in L2).
constexpr size_t STEPS_SMEM = 220 * 1024;
static size_t steps_smem(const MlpDims &d, int g_shared) {
    return mlp_shared_at64(d) + (mlp_shared_doubles(d) + (g_shared ? d.np : 0)) * sizeof(double);
}

void mlp_create(Mlp &net, int in, int out, uint64_t seed) {
    RP_REQUIRE(in >= 1 && in <= 256 && out >= 1 && out <= 8, -2, "MLP dims: in 1..256, out 1..8");
    net.in = in;
    net.out = out;
    net.np = mlp_num_params(in, out);
    std::vector<float> p(net.np, 0.f);
    // Glorot-uniform weights from a splitmix64 stream, zero biases
    uint64_t st = seed * 0x9E3779B97F4A7C15ull + 1;
    auto rnd = [&]() {
        st += 0x9E3779B97F4A7C15ull;
        uint64_t z = st;
        z = (z ^ (z >> 30)) * 0xBF58476D1CE4E5B9ull;
        z = (z ^ (z >> 27)) * 0x94D049BB133111EBull;
        z ^= z >> 31;
        return (double)(z >> 11) / 9007199254740992.0;
    };
    const MlpDims d = dims(in, out);
    auto fill = [&](int off, int rows, int cols) {
        const double a = std::sqrt(6.0 / (rows + cols));
        for (int k = 0; k < rows * cols; k++) p[off + k] = (float)((2 * rnd() - 1) * a);
    };
    fill(d.oW1, HID, in);
    fill(d.oW2, HID, HID);
    fill(d.oW3, out, HID);
    RP_CUDA(cudaMalloc((void **)&net.params, net.np * sizeof(float)));
    RP_CUDA(cudaMalloc((void **)&net.m, net.np * sizeof(float)));
    RP_CUDA(cudaMalloc((void **)&net.v, net.np * sizeof(float)));
    RP_CUDA(cudaMalloc((void **)&net.g, net.np * sizeof(float)));
    RP_CUDA(cudaMemcpy(net.params, p.data(), net.np * sizeof(float), cudaMemcpyHostToDevice));
    RP_CUDA(cudaMemset(net.m, 0, net.np * sizeof(float)));
    RP_CUDA(cudaMemset(net.v, 0, net.np * sizeof(float)));
    net.step = 0;
    // for any network: a smaller one made later must not lower the limit of those
    // before it
    const MlpDims most = dims(256, 8);
    RP_CUDA(cudaFuncSetAttribute(k_mlp_steps, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)STEPS_SMEM));
    RP_CUDA(cudaFuncSetAttribute(k_mlp_forward, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)fwd_smem(most)));
}

void mlp_free(Mlp &net) {
    if (net.params) cudaFree(net.params);
    if (net.m) cudaFree(net.m);
    if (net.v) cudaFree(net.v);
    if (net.g) cudaFree(net.g);
    if (net.io) cudaFree(net.io);
    net = Mlp{};
}

// The network's device buffer, kept between calls and grown on demand.
static char *mlp_room(Mlp &net, size_t bytes, cudaStream_t st) {
    if (bytes > net.io_cap) {
        RP_CUDA(cudaStreamSynchronize(st));
        if (net.io) cudaFree(net.io);
        net.io = nullptr;
        net.io_cap = 0;
        RP_CUDA(cudaMalloc((void **)&net.io, bytes));
        net.io_cap = bytes;
    }
    return net.io;
}

void mlp_forward(Mlp &net, const float *X_host, int n, float *Y_host, cudaStream_t st) {
    const MlpDims d = dims(net.in, net.out);
    float *dX = reinterpret_cast<float *>(mlp_room(net, (size_t)n * (d.in + d.out) * sizeof(float), st));
    float *dY = dX + (size_t)n * d.in;
    RP_CUDA(cudaMemcpyAsync(dX, X_host, (size_t)n * d.in * sizeof(float), cudaMemcpyHostToDevice, st));
    const int grid = std::min(std::max((n + MS - 1) / MS, 1), 4 * num_sms());
    k_mlp_forward<<<grid, MT, fwd_smem(d), st>>>(d, net.params, dX, n, dY);
    RP_CUDA(cudaGetLastError());
    RP_CUDA(cudaMemcpyAsync(Y_host, dY, (size_t)n * d.out * sizeof(float), cudaMemcpyDeviceToHost, st));
    RP_CUDA(cudaStreamSynchronize(st));
}

// Device buffers of a training call, carved out of the network's buffer.
struct MlpTrainBuffers {
    MlpSteps a{};
    int *idx = nullptr;
    int grid = 0, nsteps = 0;
};

static MlpTrainBuffers mlp_train_buffers(Mlp &net, const float *X_host, const float *Y_host, int n,
                                         int batch, cudaStream_t st) {
    const MlpDims d = dims(net.in, net.out);
    MlpTrainBuffers b;
    batch = std::min(batch, n);
    b.nsteps = (n + batch - 1) / batch;
    // a CTA per MS samples of a batch, one per SM at most (all resident); more
    // CTAs where those would have the parameters to update in several rounds
    // (us per batch, 21 inputs: batches of 256 15.4 -> 13.4, 64 21.8 -> 12.7, 8 54 ->
    // 12.4)
    b.a.parts = std::min((batch + MS - 1) / MS, num_sms());
    b.grid = std::max(b.a.parts, std::min((d.np + HID - 1) / HID, num_sms()));
    size_t at = 0;
    auto room = [&](size_t bytes) {
        const size_t r = at;
        at += (bytes + 255) & ~(size_t)255;
        return r;
    };
    const size_t oX = room((size_t)n * d.in * sizeof(float)), oY = room((size_t)n * d.out * sizeof(float));
    const size_t oi = room((size_t)n * sizeof(int)), og = room((size_t)b.a.parts * d.np * sizeof(double));
    const size_t ol = room((size_t)b.nsteps * sizeof(float)), op = room((size_t)b.a.parts * sizeof(double));
    const size_t oc = room(2 * sizeof(unsigned));
    char *p = mlp_room(net, at, st);
    b.a.X = reinterpret_cast<float *>(p + oX);
    b.a.Y = reinterpret_cast<float *>(p + oY);
    b.idx = reinterpret_cast<int *>(p + oi);
    b.a.gpart = reinterpret_cast<double *>(p + og);
    b.a.loss = reinterpret_cast<float *>(p + ol);
    b.a.lpart = reinterpret_cast<double *>(p + op);
    b.a.barrier = reinterpret_cast<unsigned *>(p + oc);
    b.a.err = b.a.barrier + 1;
    b.a.n = n;
    b.a.batch = batch;
    b.a.g_shared = (batch + b.a.parts - 1) / b.a.parts > MS && steps_smem(d, 1) <= STEPS_SMEM;
    b.a.params = net.params;
    b.a.m = net.m;
    b.a.v = net.v;
    b.a.g = net.g;
    RP_CUDA(cudaMemcpyAsync(p + oX, X_host, (size_t)n * d.in * sizeof(float), cudaMemcpyHostToDevice, st));
    RP_CUDA(cudaMemcpyAsync(p + oY, Y_host, (size_t)n * d.out * sizeof(float), cudaMemcpyHostToDevice, st));
    RP_CUDA(cudaMemsetAsync(b.a.err, 0, sizeof(unsigned), st));
    return b;
}

// Steps of one launch: its barrier counts two arrivals of every CTA per step and
// must not wrap (2^32 is 14 million steps of 148 CTAs; this many take 0.8 s).
constexpr int MAX_STEPS = 1 << 16;

static void mlp_steps_launch(Mlp &net, MlpTrainBuffers &b, cudaStream_t st) {
    MlpDims d = dims(net.in, net.out);
    RP_CUDA(cudaMemsetAsync(b.a.barrier, 0, sizeof(unsigned), st));
    void *args[] = {&d, &b.a};
    RP_CUDA(cudaLaunchCooperativeKernel((const void *)k_mlp_steps, dim3(b.grid), dim3(MT), args,
                                        steps_smem(d, b.a.g_shared), st));
}

// The batches' losses (and the error word) after the last launch.
static std::vector<float> mlp_losses(const MlpTrainBuffers &b, cudaStream_t st) {
    std::vector<float> l(b.nsteps);
    unsigned err = 0;
    RP_CUDA(cudaMemcpyAsync(l.data(), b.a.loss, l.size() * sizeof(float), cudaMemcpyDeviceToHost, st));
    RP_CUDA(cudaMemcpyAsync(&err, b.a.err, sizeof(err), cudaMemcpyDeviceToHost, st));
    RP_CUDA(cudaStreamSynchronize(st));
    RP_REQUIRE(err == 0, -5, "a device-side wait timed out in the network's training kernel");
    return l;
}

float mlp_grad(Mlp &net, const float *X_host, const float *Y_host, int n, float *grad_host,
               cudaStream_t st) {
    RP_REQUIRE(n >= 1, -2, "no samples");
    MlpTrainBuffers b = mlp_train_buffers(net, X_host, Y_host, n, n, st);
    mlp_steps_launch(net, b, st);
    const float loss = mlp_losses(b, st)[0];
    RP_CUDA(cudaMemcpy(grad_host, net.g, net.np * sizeof(float), cudaMemcpyDeviceToHost));
    return loss;
}

float mlp_train(Mlp &net, const float *X_host, const float *Y_host, int n, int epochs, int batch,
                float lr, uint64_t seed, cudaStream_t st) {
    RP_REQUIRE(n >= 1 && epochs >= 1 && batch >= 1, -2, "bad training arguments");
    MlpTrainBuffers b = mlp_train_buffers(net, X_host, Y_host, n, batch, st);
    b.a.idx = b.idx;
    b.a.update = 1;
    b.a.lr = lr;
    // one shuffle per epoch on the host (deterministic), while the device
    // still runs the epoch before
    std::vector<int> idx(n);
    for (int i = 0; i < n; i++) idx[i] = i;
    uint64_t s = seed * 6364136223846793005ull + 1442695040888963407ull;
    for (int e = 0; e < epochs; e++) {
        for (int i = n - 1; i > 0; i--) {
            s = s * 6364136223846793005ull + 1442695040888963407ull;
            const int k = (int)((s >> 33) % (uint64_t)(i + 1));
            std::swap(idx[i], idx[k]);
        }
        RP_CUDA(cudaMemcpyAsync(b.idx, idx.data(), (size_t)n * sizeof(int), cudaMemcpyHostToDevice, st));
        MlpTrainBuffers part = b;
        for (int64_t s0 = 0; s0 < b.nsteps; s0 += MAX_STEPS) {
            const int64_t at = s0 * b.a.batch;
            part.a.idx = b.a.idx + at;
            part.a.n = (int)std::min<int64_t>(n - at, (int64_t)MAX_STEPS * b.a.batch);
            part.a.loss = b.a.loss + s0;
            part.a.step0 = net.step + (int)s0;
            mlp_steps_launch(net, part, st);
        }
        net.step += b.nsteps;
    }
    double tot = 0.0;
    for (float l : mlp_losses(b, st)) tot += l;
    return (float)(tot / b.nsteps);
}

void mlp_get(Mlp &net, float *p) {
    RP_CUDA(cudaMemcpy(p, net.params, net.np * sizeof(float), cudaMemcpyDeviceToHost));
}
void mlp_set(Mlp &net, const float *p) {
    RP_CUDA(cudaMemcpy(net.params, p, net.np * sizeof(float), cudaMemcpyHostToDevice));
    RP_CUDA(cudaMemset(net.m, 0, net.np * sizeof(float)));
    RP_CUDA(cudaMemset(net.v, 0, net.np * sizeof(float)));
    net.step = 0;
}

}  // namespace rp
