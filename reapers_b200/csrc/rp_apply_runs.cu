// Run kernel: H.psi = sum_x D_x(n) psi[n ^ x], D_x(n) = sum of the
// coefficients of the terms with X mask x, signed by (-1)^popc(z & n).
//
// Used below the row kernel's size, and above it for lists too long for that
// kernel's table whose terms share X masks (plan_build has the rules).  For states
// up to 2^14 elements a term's cost is its instructions, not its bytes (the state
// sits in L1 / L2), and there are too few tiles of output to fill the GPU.  So the
// work is cut both ways: a warp owns 32 << eb output elements (lane = the low 5
// index bits, eb bits in registers) and one worker's share of the terms; the eight
// warps of `parts` CTAs are the workers of one block of outputs.  Their sums meet in
// shared memory and then in a buffer of partial sums, where the block's last CTA to
// arrive adds the parts in order (one launch, and the same bits run to run).
// Clusters in place of the buffer were slower: eight-CTA clusters left 55 of 148 SMs
// idle while others held two CTAs (dense SYK on 12 qubits 28 us, against the figures
// below).
//
// Terms with one X mask form a run: the run's diagonal factor is summed first
// and then multiplied once with the gathered elements, so the loads and
// multiply-adds are per run (dense SYK on 12 qubits: 10626 terms, 794 runs).  The signs cost no population count per
// term and warp: 32 terms at a time, lane k folds term k's parity over the
// block's index bits into its coefficient and expands the lane and register
// parts of its Z mask into 32-bit and 8-bit sign masks, which the whole warp
// then reads back from shared memory.
//
// Bound by instruction issue (the adds and sign flips of the factors) and, on
// small states, by the launch and the latency of a few dependent loads.
// Measured, us per product, tiled kernel (a thread per element, terms in a row)
// -> this one: dense SYK, 12 qubits complex128 2285 -> 18.6, complex64 2315 ->
// 15.6; 14 qubits complex128 8780 -> 92; sparse SYK, 14 qubits complex64 87 ->
// 8.6, 16 qubits 101 -> 18.6; XXZ chain, 16 qubits complex128 26 -> 6.5; dense SYK, 18
// qubits complex64 (58905 terms, 3214 masks) 27.5 -> 2.7 ms, 20 qubits 72 -> 16, 22 qubits
// 375 -> 94.
// Summing a run's terms by buckets of equal register signs and a Walsh-Hadamard
// transform took fewer instructions but was a longer chain: 35 -> 70 us.
#include <algorithm>

#include "rp_apply.cuh"
#include "rp_apply_runs.cuh"

namespace rp {

constexpr int RUN_W = 8;                 // warps (workers) per CTA
constexpr int RUN_T = 32 * RUN_W;

template <typename Real>
struct RunArgs {
    const Cplx<Real> *in;
    Cplx<Real> *out;
    const RunTerm *terms;
    const Run *runs;
    const uint32_t *wstart;
    Cplx<Real> *partial;                 // [part][element]
    unsigned *arrived;                   // per block, 0 between launches
    int parts;
    int span;                            // planned workers' shares that a warp takes
    size_t dim;
    double alpha;
    const double *alpha_dev;
    int accumulate;
    const int *active;
};

// A staged term: the coefficient's bits, the lane sign mask and the register
// sign mask (bit e set: negative for register element e).
struct alignas(16) StagedTerm {
    uint32_t lo, hi, lane_mask, reg_mask;
};

template <typename Real>
__device__ __forceinline__ Real staged_coeff(const StagedTerm &s, uint32_t flip);
template <>
__device__ __forceinline__ double staged_coeff<double>(const StagedTerm &s, uint32_t flip) {
    return __hiloint2double((int)(s.hi ^ flip), (int)s.lo);
}
template <>
__device__ __forceinline__ float staged_coeff<float>(const StagedTerm &s, uint32_t flip) {
    return __uint_as_float(s.hi ^ flip);
}

// c negated where bit 31 of s is set.
__device__ __forceinline__ double flip_if(double c, uint32_t s) {
    return __hiloint2double(__double2hiint(c) ^ (int)(s & 0x80000000u), __double2loint(c));
}
__device__ __forceinline__ float flip_if(float c, uint32_t s) {
    return __uint_as_float(__float_as_uint(c) ^ (s & 0x80000000u));
}

// A load that takes other CTAs' stores from L2.
__device__ __forceinline__ Cplx<double> ld_l2(const Cplx<double> *p) {
    const double2 v = __ldcg(reinterpret_cast<const double2 *>(p));
    return {v.x, v.y};
}
__device__ __forceinline__ Cplx<float> ld_l2(const Cplx<float> *p) {
    const float2 v = __ldcg(reinterpret_cast<const float2 *>(p));
    return {v.x, v.y};
}

template <typename Real, int EB>
__global__ void __launch_bounds__(RUN_T, 2) k_apply_runs(const RunArgs<Real> a) {
    constexpr int E = 1 << EB;
    constexpr int N = 32 * E;            // output elements of a block
    __shared__ StagedTerm staged[RUN_W][32];
    __shared__ Cplx<Real> part[RUN_W][N];
    __shared__ bool s_last;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    const unsigned rank = blockIdx.x % (unsigned)a.parts;
    const uint32_t block = blockIdx.x / (unsigned)a.parts;
    const int worker = ((int)rank * RUN_W + warp) * a.span;
    const uint32_t r1 = a.wstart[worker + a.span];
    uint32_t r = a.wstart[worker];
    Cplx<Real> acc[E];
#pragma unroll
    for (int e = 0; e < E; e++) acc[e].x = acc[e].y = Real(0);
    // terms of a worker are contiguous: [k, kend) by batches of 32
    uint32_t k = 0, batch = 0, kend = 0;
    if (r < r1) {
        const Run last = a.runs[r1 - 1];
        k = batch = a.runs[r].first;
        kend = last.first + last.nr + last.ni;
    }
    RunTerm ahead{};                     // this lane's term of the next batch
    if (batch + lane < kend) ahead = a.terms[batch + lane];
    auto stage = [&] {
        __syncwarp();
        if (batch + lane < kend) {
            const RunTerm t = ahead;
            double c = (__popc((t.z >> (5 + EB)) & block) & 1) ? -t.c : t.c;
            StagedTerm s;
            if constexpr (sizeof(Real) == 8) {
                s.lo = (uint32_t)__double2loint(c);
                s.hi = (uint32_t)__double2hiint(c);
            } else {
                s.lo = 0u;
                s.hi = __float_as_uint((float)c);
            }
            s.lane_mask = (t.z & 1u ? 0xAAAAAAAAu : 0u) ^ (t.z & 2u ? 0xCCCCCCCCu : 0u) ^
                          (t.z & 4u ? 0xF0F0F0F0u : 0u) ^ (t.z & 8u ? 0xFF00FF00u : 0u) ^
                          (t.z & 16u ? 0xFFFF0000u : 0u);
            const uint32_t zr = (t.z >> 5) & (uint32_t)(E - 1);
            s.reg_mask = (zr & 1u ? 0xAAu : 0u) ^ (zr & 2u ? 0xCCu : 0u) ^ (zr & 4u ? 0xF0u : 0u);
            staged[warp][lane] = s;
        }
        batch += 32;
        if (batch + lane < kend) ahead = a.terms[batch + lane];
        __syncwarp();
    };
    // d[e] = sum of the n terms from k on, signed for element e of this lane
    auto factor = [&](Real(&d)[E], uint32_t n) {
#pragma unroll
        for (int e = 0; e < E; e++) d[e] = Real(0);
        while (n) {
            if (k == batch) stage();
            const StagedTerm *s = &staged[warp][k - (batch - 32u)];
            const uint32_t m = min(n, batch - k);
#pragma unroll 4
            for (uint32_t i = 0; i < m; i++) {
                const StagedTerm t = s[i];
                const Real c = staged_coeff<Real>(t, (t.lane_mask >> lane) << 31);
#pragma unroll
                for (int e = 0; e < E; e++) d[e] += flip_if(c, t.reg_mask << (31 - e));
            }
            k += m;
            n -= m;
        }
    };
    Run run{};
    if (r < r1) run = a.runs[r];
    wait_prior_kernel();
    if (a.active && *a.active == 0) return;   // the same in every CTA
    while (r < r1) {
        const uint32_t xl = run.x & 31u, xe = (run.x >> 5) & (uint32_t)(E - 1);
        const Cplx<Real> *src = a.in + ((size_t)(block ^ (run.x >> (5 + EB))) * N + (lane ^ xl));
        Cplx<Real> v[E];
#pragma unroll
        for (int e = 0; e < E; e++) v[e] = src[(e ^ xe) << 5];
        const Run cur = run;
        if (++r < r1) run = a.runs[r];
        Real d[E];
        if (cur.nr) {
            factor(d, cur.nr);
#pragma unroll
            for (int e = 0; e < E; e++) {
                acc[e].x = fma(d[e], v[e].x, acc[e].x);
                acc[e].y = fma(d[e], v[e].y, acc[e].y);
            }
        }
        if (cur.ni) {
            factor(d, cur.ni);
#pragma unroll
            for (int e = 0; e < E; e++) {
                acc[e].x = fma(-d[e], v[e].y, acc[e].x);
                acc[e].y = fma(d[e], v[e].x, acc[e].y);
            }
        }
    }
    // the CTA's workers in order, then the block's parts in order
#pragma unroll
    for (int e = 0; e < E; e++) part[warp][(e << 5) | lane] = acc[e];
    __syncthreads();
    const double scale = a.alpha * (a.alpha_dev ? *a.alpha_dev : 1.0);
    auto store = [&](int i, Cplx<Real> s) {
        Cplx<Real> *p = a.out + (size_t)block * N + i;
        s.x = (Real)(scale * (double)s.x);
        s.y = (Real)(scale * (double)s.y);
        if (a.accumulate) {
            const Cplx<Real> old = *p;
            s.x += old.x;
            s.y += old.y;
        }
        *p = s;
    };
    if (threadIdx.x < N) {
        Cplx<Real> s = part[0][threadIdx.x];
#pragma unroll
        for (int w = 1; w < RUN_W; w++) {
            s.x += part[w][threadIdx.x].x;
            s.y += part[w][threadIdx.x].y;
        }
        if (a.parts == 1) store(threadIdx.x, s);
        else a.partial[rank * a.dim + (size_t)block * N + threadIdx.x] = s;
    }
    if (a.parts == 1) return;
    __threadfence();
    __syncthreads();
    // atomicInc wraps to 0 with the last arrival: ready for the next launch
    if (threadIdx.x == 0) s_last = atomicInc(&a.arrived[block], a.parts - 1) == (unsigned)a.parts - 1;
    __syncthreads();
    if (!s_last) return;
    __threadfence();
    if (threadIdx.x < N) {
        Cplx<Real> s{Real(0), Real(0)};
        const Cplx<Real> *q = a.partial + (size_t)block * N + threadIdx.x;
#pragma unroll 4
        for (int c = 0; c < a.parts; c++) {
            const Cplx<Real> v = ld_l2(q + c * a.dim);
            s.x += v.x;
            s.y += v.y;
        }
        store(threadIdx.x, s);
    }
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------

// Cost of a run and of a term in it, in issue slots of a warp (8 elements per
// lane); only their ratio matters to the split.
constexpr double RUN_COST = 70.0, TERM_COST = 32.0;
// A worker's least share: below it, another part costs more (the exchange
// through L2) than it takes off.
constexpr double MIN_SHARE = 400.0;
constexpr int MAX_PARTS = 32;

void runplan_build(RunPlan &p, int len, const uint64_t *bits, const double *coeff, int64_t nterms) {
    p = RunPlan{};
    if (len < RUN_MIN_LEN || nterms < 1) return;
    struct T {
        uint32_t x, z;
        double c;
        int kind;
    };
    std::vector<T> ts;
    ts.reserve(nterms);
    for (int64_t k = 0; k < nterms; k++) {
        const uint32_t x = even_bits(bits[k]), z = even_bits(bits[k] >> 1);
        // the sign rule takes the source index n ^ x
        const double s = (__builtin_popcount(z & x) & 1) ? -1.0 : 1.0;
        const double cr = coeff[2 * k], ci = coeff[2 * k + 1];
        if (cr != 0.0 || ci == 0.0) ts.push_back({x, z, s * cr, 0});
        if (ci != 0.0) ts.push_back({x, z, s * ci, 1});
    }
    // by mask, then kind of coefficient, in the list's order among equals: a byte of
    // the key at a time, least significant first
    std::vector<T> other(ts.size());
    for (int shift = 0; shift <= len; shift += 8) {
        auto digit = [shift](const T &t) { return (((uint64_t)t.x << 1 | (uint64_t)t.kind) >> shift) & 255u; };
        size_t at[257] = {};
        for (const T &t : ts) at[digit(t) + 1]++;
        for (int d = 0; d < 256; d++) at[d + 1] += at[d];
        for (const T &t : ts) other[at[digit(t)]++] = t;
        ts.swap(other);
    }
    p.eb = std::min(3, len - 5);
    double total = 0.0;
    for (size_t k = 0; k < ts.size(); k++)
        total += TERM_COST + (k == 0 || ts[k].x != ts[k - 1].x ? RUN_COST : 0.0);
    p.nblocks = 1 << (len - 5 - p.eb);
    // as many parts per block of outputs as fill the GPU with two CTAs per SM,
    // if each worker keeps its least share
    p.parts = std::min({MAX_PARTS, 2 * num_sms() / p.nblocks, (int)(total / (MIN_SHARE * RUN_W))});
    p.parts = std::max(p.parts, 1);
    const int workers = p.parts * RUN_W;
    p.terms.reserve(ts.size());
    // contiguous shares of equal cost; a run cut by a boundary continues as
    // another run of the next worker
    p.wstart.assign(1, 0u);
    double load = 0.0, rest = total;   // this worker's so far; what is not dealt out
    for (size_t k = 0; k < ts.size(); k++) {
        bool fresh = k == 0 || ts[k].x != ts[k - 1].x;
        const double next = TERM_COST + (fresh ? RUN_COST : 0.0);
        const int left = workers - (int)p.wstart.size() + 1;   // this worker and those after
        rest -= next;
        if (left > 1 && load > 0.0 && load + 0.5 * next >= (load + next + rest) / left) {
            load = 0.0;
            p.wstart.push_back((uint32_t)p.runs.size());
            fresh = true;
        }
        if (fresh) p.runs.push_back({ts[k].x, (uint32_t)k, 0u, 0u});
        load += TERM_COST + (fresh ? RUN_COST : 0.0);
        (ts[k].kind ? p.runs.back().ni : p.runs.back().nr)++;
        p.terms.push_back({ts[k].c, ts[k].z, 0u});
    }
    while ((int)p.wstart.size() <= workers) p.wstart.push_back((uint32_t)p.runs.size());
    p.ok = true;
}

// Partial sums and arrival counts of blocks that several CTAs share: one buffer for
// all plans, whose launches run one after the other on the library's stream (captured
// ones do without it).  Shared blocks have at most two CTAs per SM in all, so its size
// is fixed; a buffer per plan cost 0.37 ms of a plan's creation.
static char *g_runs = nullptr;

static size_t runs_partial_bytes() { return (size_t)2 * num_sms() * 256 * sizeof(Cplx<double>); }

static char *runs_scratch() {
    if (g_runs) return g_runs;
    const size_t count = (size_t)2 * num_sms() * sizeof(unsigned);
    void *p = nullptr;
    RP_CUDA(cudaMalloc(&p, runs_partial_bytes() + count));
    g_runs = static_cast<char *>(p);
    RP_CUDA(cudaMemset(g_runs + runs_partial_bytes(), 0, count));
    return g_runs;
}

void runs_scratch_release() {
    if (g_runs) cudaFree(g_runs);
    g_runs = nullptr;
}

void runplan_upload(RunPlan &p) {
    if (!p.ok) return;
    runplan_free(p);
    TablePack t;
    t.add(p.terms);
    p.at_runs = t.add(p.runs);
    p.at_wstart = t.add(p.wstart);
    p.dev = t.upload();
    if (p.parts > 1) runs_scratch();
}

void runplan_free(RunPlan &p) {
    if (p.dev) cudaFree(p.dev);
    p.dev = nullptr;
}

template <typename Real, int EB>
static void launch_runs(const RunPlan &p, const RunLaunch &l, cudaStream_t st) {
    RunArgs<Real> a;
    a.in = static_cast<const Cplx<Real> *>(l.in);
    a.out = static_cast<Cplx<Real> *>(l.out);
    a.terms = reinterpret_cast<const RunTerm *>(p.dev);
    a.runs = reinterpret_cast<const Run *>(p.dev + p.at_runs);
    a.wstart = reinterpret_cast<const uint32_t *>(p.dev + p.at_wstart);
    // Captured products keep no partial sums: replays of two graphs may overlap, on
    // other streams than the library's, and would share the buffer.  One CTA
    // then takes all parts of its block, us outside / inside a graph / tiled kernel there:
    // sparse SYK, complex128, 12 qubits 6.1 / 10.2 / 49, 14 qubits 7.5 / 11.7 / 86; dense SYK,
    // 8 qubits 6.6 / 29 / 377, 12 qubits 16.7 / 117 / 2283.
    cudaStreamCaptureStatus capture = cudaStreamCaptureStatusNone;
    if (p.parts > 1) RP_CUDA(cudaStreamIsCapturing(st, &capture));
    a.span = capture == cudaStreamCaptureStatusNone ? 1 : p.parts;
    a.parts = p.parts / a.span;
    char *const shared = a.parts > 1 ? runs_scratch() : nullptr;
    a.partial = reinterpret_cast<Cplx<Real> *>(shared);
    a.arrived = shared ? reinterpret_cast<unsigned *>(shared + runs_partial_bytes()) : nullptr;
    a.dim = (size_t)p.nblocks * (32u << EB);
    a.alpha = l.alpha;
    a.alpha_dev = l.alpha_dev;
    a.accumulate = l.accumulate;
    a.active = l.active;
    launch_dependent(k_apply_runs<Real, EB>, p.nblocks * a.parts, RUN_T, 0, st, 1, a);
}

template <typename Real>
static void launch_runs_eb(const RunPlan &p, const RunLaunch &l, cudaStream_t st) {
    switch (p.eb) {
    case 0: launch_runs<Real, 0>(p, l, st); break;
    case 1: launch_runs<Real, 1>(p, l, st); break;
    case 2: launch_runs<Real, 2>(p, l, st); break;
    default: launch_runs<Real, 3>(p, l, st); break;
    }
}

void runs_launch(const RunPlan &p, int dtype, const RunLaunch &l, cudaStream_t st) {
    RP_REQUIRE(p.ok, -2, "run kernel not planned for this Hamiltonian");
    if (dtype == 2) launch_runs_eb<double>(p, l, st);
    else launch_runs_eb<float>(p, l, st);
}

}  // namespace rp
