// Restarted Krylov exp(-(beta + i t) H) psi (Eiermann-Ernst), GPU-resident.
//
// Control flow follows Krylov::evolve / arnoldi / orthogonalize of the
// reference (inc/algo.h:77-173, 267-365) step for step -- the same pass
// criterion (eta = 1/sqrt 2, at most three passes, first comparison against
// eta/2), the same breakdown rule, the same growing block Hessenberg matrix
// and the same convergence test on ||Hexp0|| -- so the number of H.psi
// products and restarts match the reference.  What differs is how each step
// touches HBM:
//   * projections of a pass are taken all at once (classical Gram-Schmidt
//     per pass) instead of one inner product + axpy per basis vector;
//   * the update w -= sum h_i v_i and ||w|| are one fused pass, and a step's
//     passes, with their decisions, one cooperative launch (rp_kry_ortho.cu);
//   * the basis is stored unnormalised with per-vector scale factors, so no
//     normalisation pass is made;
//   * all decisions are taken on the device, so a whole Arnoldi cycle is
//     enqueued without a host round trip, and the host synchronises once per
//     restart.
// Inner products, norms, H, Hfull and its exponential are FP64 on the GPU for
// both vector precisions.
#include <algorithm>
#include <cmath>
#include <cstdlib>
#include <cstring>

#include "rp_expm_impl.cuh"
#include "rp_krylov.cuh"

namespace rp {

static size_t esize(int dtype) { return dtype == 2 ? 16 : 8; }

// The first orthogonalisation pass's projections <v_i|w> can be taken in the
// H.psi kernel's epilogue (w never leaves the SM before it is projected) or by
// the grouped projection kernel after the apply.  The separate kernel streams
// the basis at a higher fraction of HBM bandwidth than the epilogue, whose
// per-row warp reductions slow the apply, so it is the default;
// RPB200_FUSED_DOTS=1 selects the fused form.
static bool fused_projections() {
    static int v = -1;
    if (v < 0) {
        const char *e = getenv("RPB200_FUSED_DOTS");
        v = (e && e[0] == '1') ? 1 : 0;
    }
    return v == 1;
}

void workspace_matrix(KryWorkspace &ws, int need, cudaStream_t st) {
    if (need <= ws.hcap) return;
    int cap = std::max(ws.hcap ? ws.hcap : 4 * ws.krydim, 32);
    while (cap < need) cap *= 2;
    // both before either is replaced: a workspace without room stays as it is
    void *nh = nullptr, *ns = nullptr;
    if (cudaMalloc(&nh, (size_t)cap * cap * sizeof(cd)) != cudaSuccess ||
        cudaMalloc(&ns, ((size_t)2 * cap * cap + expm_scratch_elems(cap)) * sizeof(cd)) != cudaSuccess) {
        cudaGetLastError();
        if (nh) cudaFree(nh);
        throw Error{-4, "device out of memory for the Krylov matrix of " + std::to_string(need) + " rows"};
    }
    RP_CUDA(cudaMemsetAsync(nh, 0, (size_t)cap * cap * sizeof(cd), st));
    if (ws.hfull) {
        RP_CUDA(cudaMemcpy2DAsync(nh, (size_t)cap * sizeof(cd), ws.hfull,
                                  (size_t)ws.hcap * sizeof(cd), (size_t)ws.hcap * sizeof(cd),
                                  ws.hcap, cudaMemcpyDeviceToDevice, st));
        RP_CUDA(cudaStreamSynchronize(st));
        cudaFree(ws.hfull);
    }
    if (ws.escratch) cudaFree(ws.escratch);
    ws.hfull = nh;
    ws.escratch = ns;
    ws.hcap = cap;
}

void workspace_release(KryWorkspace &ws) {
    for (void *p : ws.mem) cudaFree(p);
    if (ws.hfull) cudaFree(ws.hfull);
    if (ws.escratch) cudaFree(ws.escratch);
    ws = KryWorkspace{};
}

// `bytes` more of device memory for the workspace, or nothing.
static char *workspace_more(KryWorkspace &ws, size_t bytes) {
    void *p = nullptr;
    if (cudaMalloc(&p, bytes) != cudaSuccess) {
        cudaGetLastError();
        throw Error{-4, "device out of memory for the Krylov workspace (" + std::to_string(bytes) + " bytes)"};
    }
    ws.mem.push_back(p);
    return static_cast<char *>(p);
}

// One allocation for all vectors (one each took 0.3 ms at 8 MB) and the small state.
void workspace_ensure(KryWorkspace &ws, int len, int dtype, int krydim) {
    const size_t vb = (((size_t)esize(dtype) << len) + 255) & ~(size_t)255;
    if (ws.dev && ws.len == len && ws.dtype == dtype) {
        if (krydim <= ws.krydim) return;
        // a larger basis for the same state: add vectors, keep the rest (as they
        // were, when there is no room)
        char *p = workspace_more(ws, (size_t)(krydim - ws.krydim) * vb);
        for (; ws.krydim < krydim; ws.krydim++, p += vb) ws.u.push_back(p);
        return;
    }
    workspace_release(ws);
    const int g = std::max(num_sms(), reduce_grid());
    size_t at = (size_t)(krydim + 2) * vb;
    auto room = [&](size_t bytes) {
        const size_t r = at;
        at += (bytes + 255) & ~(size_t)255;
        return r;
    };
    const size_t o_dev = room(sizeof(KryDev)), o_part = room((size_t)g * (MAX_KRYLOV + 1) * 2 * sizeof(double));
    const size_t o_norm = room((size_t)g * sizeof(double)), o_err = room(sizeof(unsigned));
    const size_t o_tab = room((MAX_KRYLOV + 1) * sizeof(void *));
    char *p = workspace_more(ws, at);
    ws.len = len;
    ws.dtype = dtype;
    ws.krydim = krydim;
    ws.D = 1ull << len;
    for (int i = 0; i <= krydim; i++) ws.u.push_back(p + (size_t)i * vb);
    ws.y = p + (size_t)(krydim + 1) * vb;
    ws.dev = reinterpret_cast<KryDev *>(p + o_dev);
    ws.partials = reinterpret_cast<double *>(p + o_part);
    ws.norm_partials = reinterpret_cast<double *>(p + o_norm);
    ws.err = reinterpret_cast<unsigned *>(p + o_err);
    ws.tab = reinterpret_cast<void **>(p + o_tab);
    RP_CUDA(cudaMemset(ws.err, 0, sizeof(unsigned)));
}

// ---------------------------------------------------------------------------
// Control kernels (one CTA each; they only touch the small state)
// ---------------------------------------------------------------------------
__global__ void k_kry_init(KryDev *s, double beta0) {
    if (threadIdx.x == 0) {
        memset(s, 0, offsetof(KryDev, sigma));
        s->beta0 = beta0;
        s->sigma[0] = 1.0 / beta0;
    }
}

__global__ void k_kry_begin(KryDev *s, int krydim, int restart) {
    if (threadIdx.x == 0) {
        s->active = 1;
        s->barrier = 0;
        s->m_eff = krydim;
        s->brokedown = 0;
        if (restart) {
            // the last basis vector v_m is the next starting vector
            s->sigma[0] = s->sigma[krydim];
            s->oldbeta = s->beta;
        }
    }
    for (int i = threadIdx.x; i < 2 * krydim * krydim; i += blockDim.x) s->H[i] = 0.0;
}

// Grow Hfull by the cycle's block (Algorithm 2 of Eiermann & Ernst, as in
// inc/algo.h:303-328), take column 0 of exp(f * Hfull) (f = -(t_imag + i
// t_real)), its last m entries (Hexp0), their norm, and the update
// coefficients beta0 * Hexp0_i * sigma_i.  in_smem: Hfull's blocks fit in
// shared memory beside the three vectors (else they go to scratch).
__global__ void __launch_bounds__(768) k_kry_expm(KryDev *s, cd *hfull, int hcap, cd *scratch,
                                                   int krydim, int cycle, double fr, double fi,
                                                   int in_smem, int action, const unsigned *err) {
    extern __shared__ __align__(16) unsigned char expm_smem[];
    if (threadIdx.x == 0) s->err = *err;
    const int m = s->m_eff;
    const int base = (cycle - 1) * krydim;
    const int n = base + m;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e % n, j = e / n;
        if (i >= base || j >= base) hfull[i + (size_t)j * hcap] = cd{0.0, 0.0};
    }
    __syncthreads();
    if (threadIdx.x == 0 && cycle > 1) hfull[base + (size_t)(base - 1) * hcap] = cd{s->oldbeta, 0.0};
    for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
        const int i = e % m, j = e / m;
        hfull[(base + i) + (size_t)(base + j) * hcap] =
            cd{s->H[2 * (i + j * krydim)], s->H[2 * (i + j * krydim) + 1]};
    }
    __syncthreads();
    const cd f{fr, fi};
    cd *col = nullptr;
    if (action) {
        const int N = cycle * krydim;
        cd *const v = reinterpret_cast<cd *>(expm_smem), *const w = v + N, *const y = w + N;
        cd *const sub = y + N, *const blk = in_smem ? sub + cycle : scratch;
        for (int e = threadIdx.x; e < cycle * krydim * krydim; e += blockDim.x) {
            const int b = e / (krydim * krydim), i = e % krydim, j = e / krydim % krydim;
            const int r = b * krydim + i, c = b * krydim + j;
            if (r < n && c < n) blk[((size_t)b * krydim + i) * krydim + j] = hfull[r + (size_t)c * hcap];
        }
        for (int b = threadIdx.x; b < cycle; b += blockDim.x)
            sub[b] = b ? hfull[b * krydim + (size_t)(b * krydim - 1) * hcap] : cd{0.0, 0.0};
        __syncthreads();
        if (expm_action(ActionMatrix{blk, sub, krydim, cycle, m, true}, f, v, w, y)) col = y;
    }
    if (!col) {
        cd *A = scratch, *E = scratch + (size_t)n * n, *ws = E + (size_t)n * n;
        for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
            const int i = e % n, j = e / n;
            A[e] = cmul(f, hfull[i + (size_t)j * hcap]);
        }
        __syncthreads();
        expm_block(n, A, E, ws, reinterpret_cast<double *>(expm_smem));
        col = E;
    }
    if (threadIdx.x == 0) {
        double sq = 0.0;
        for (int i = 0; i < m; i++) {
            const cd e = col[base + i];
            sq += e.x * e.x + e.y * e.y;
        }
        s->nrm = sqrt(sq);
    }
    for (int i = threadIdx.x; i < m; i += blockDim.x) {
        const cd e = col[base + i];
        const double c = s->beta0 * s->sigma[i];
        s->ycoef[2 * i] = c * e.x;
        s->ycoef[2 * i + 1] = c * e.y;
    }
}

// Shared memory of the exponential kernels: what a CTA can have at most.
constexpr size_t EXPM_SMEM = 200 * 1024;

static void kry_expm_launch(KryWorkspace &ws, int krydim, int cycle, double fr, double fi, cudaStream_t st) {
    const size_t n = (size_t)cycle * krydim;
    const size_t vecs = (3 * n + cycle) * sizeof(cd), blocks = n * krydim * sizeof(cd);
    const size_t pade = (2 * n + 64) * sizeof(double);
    const int action = vecs <= EXPM_SMEM, in_smem = vecs + blocks <= EXPM_SMEM;
    const size_t smem = std::max(pade, in_smem ? vecs + blocks : action ? vecs : 0);
    // always the same value: without it a request just below 48 KB fails too, the
    // kernel's own static variables counting towards that limit
    RP_CUDA(cudaFuncSetAttribute(k_kry_expm, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)EXPM_SMEM));
    k_kry_expm<<<1, 768, smem, st>>>(ws.dev, (cd *)ws.hfull, ws.hcap, (cd *)ws.escratch, krydim, cycle, fr,
                                      fi, in_smem, action, ws.err);
    RP_CUDA(cudaGetLastError());
}

// The first `bytes` of a device state in pinned host memory, the stream being
// idle afterwards: one copy for all that a call reads back.
static KryDev *g_host = nullptr;

static const KryDev &read_back(const KryDev *dev, size_t bytes, cudaStream_t st) {
    if (!g_host) RP_CUDA(cudaHostAlloc((void **)&g_host, sizeof(KryDev), cudaHostAllocDefault));
    RP_CUDA(cudaMemcpyAsync(g_host, dev, bytes, cudaMemcpyDeviceToHost, st));
    RP_CUDA(cudaStreamSynchronize(st));
    RP_REQUIRE(g_host->err == 0, -5, "a device-side wait timed out in the H.psi kernel");
    return *g_host;
}

// Device state of the Lanczos steps and combinations over the caller's vectors:
// fixed, and apart from the workspace, whose basis they leave alone.
struct LanczosScratch {
    KryDev *dev = nullptr;
    double *partials = nullptr;          // two sums per CTA
    unsigned *err = nullptr;
};
static LanczosScratch g_lan;

static const LanczosScratch &lanczos_scratch() {
    if (g_lan.dev) return g_lan;
    const size_t at = (sizeof(KryDev) + 15) & ~(size_t)15, pb = (size_t)reduce_grid() * 2 * sizeof(double);
    char *p = nullptr;
    if (cudaMalloc((void **)&p, at + pb + sizeof(unsigned)) != cudaSuccess) {
        cudaGetLastError();
        throw Error{-4, "device out of memory for the Lanczos scratch"};
    }
    g_lan.dev = reinterpret_cast<KryDev *>(p);
    g_lan.partials = reinterpret_cast<double *>(p + at);
    g_lan.err = reinterpret_cast<unsigned *>(p + at + pb);
    return g_lan;
}

void krylov_scratch_release() {
    if (g_host) cudaFreeHost(g_host);
    g_host = nullptr;
    if (g_lan.dev) cudaFree(g_lan.dev);
    g_lan = LanczosScratch{};
}

__global__ void k_kry_err(KryDev *s, const unsigned *err) { s->err = *err; }

// One Arnoldi cycle: m products and orthogonalisation steps, enqueued without
// a host round trip (a breakdown switches the rest off on the device).
static void arnoldi_cycle(const ApplyPlan &plan, KryWorkspace &ws, int m, bool restart, cudaStream_t st) {
    KryDev *s = ws.dev;
    k_kry_begin<<<1, 256, 0, st>>>(s, m, restart);
    RP_CUDA(cudaGetLastError());
    VecTable tab{};
    for (int i = 0; i <= m; i++) tab.p[i] = ws.u[i];
    const bool fused = apply_fuses_dots(plan) && fused_projections();
    if (fused)   // the pointer table on the device, for the product's epilogue
        RP_CUDA(cudaMemcpyAsync(ws.tab, tab.p, (m + 1) * sizeof(void *), cudaMemcpyHostToDevice, st));
    for (int j = 0; j < m; j++) {
        ApplyLaunch L;
        L.in = ws.u[j];
        L.out = ws.u[j + 1];
        L.alpha_dev = &s->sigma[j];
        L.active = &s->active;
        L.err = ws.err;
        if (fused) {
            L.dot_vecs = (const void *const *)ws.tab;
            L.ndot = j + 1;
            L.partials = ws.partials;
        }
        apply_launch(plan, L, st);
        ortho_launch(plan.dtype, ws.D, tab, ws.u[j + 1], s, ws.partials, ws.norm_partials, ws.err, j, m,
                     fused ? apply_grid(plan) : 0, st);
    }
}

void krylov_evolve(const ApplyPlan &plan, KryWorkspace &ws, void *psi, double t_real,
                   double t_imag, int krydim, double tol, int max_iters, EvolveStats *stats,
                   cudaStream_t st) {
    RP_REQUIRE(krydim >= 2 && krydim <= MAX_KRYLOV, -2, "krydim must be in [2, 64]");
    RP_REQUIRE(psi, -2, "null state vector");
    EvolveStats S{};
    if (stats) *stats = S;
    // State::evolve returns immediately for t == 0 and beta == 0 (inc/state.h:418)
    if (t_real == 0.0 && t_imag == 0.0) return;
    workspace_ensure(ws, plan.len, plan.dtype, krydim);
    const uint64_t D = ws.D;
    const int dtype = plan.dtype;
    const double beta0 = vec_norm(dtype, D, psi, st);
    if (beta0 == 0.0) return;   // exp(A) 0 = 0
    RP_CUDA(cudaMemcpyAsync(ws.u[0], psi, D * esize(dtype), cudaMemcpyDeviceToDevice, st));
    RP_CUDA(cudaMemsetAsync(ws.y, 0, D * esize(dtype), st));
    RP_CUDA(cudaMemsetAsync(ws.err, 0, sizeof(unsigned), st));
    k_kry_init<<<1, 32, 0, st>>>(ws.dev, beta0);
    RP_CUDA(cudaGetLastError());

    KryDev *s = ws.dev;
    int cycle = 0;
    KryDev const *hdr = nullptr;
    while (true) {
        cycle++;
        workspace_matrix(ws, cycle * krydim, st);
        arnoldi_cycle(plan, ws, krydim, cycle > 1, st);
        VecTable tab{};
        for (int i = 0; i <= krydim; i++) tab.p[i] = ws.u[i];
        kry_expm_launch(ws, krydim, cycle, -t_imag, -t_real, st);
        multi_axpy(dtype, D, tab, krydim, &s->m_eff, s->ycoef, ws.y, st);
        hdr = &read_back(s, offsetof(KryDev, sigma), st);
        S.restarts = cycle;
        S.applies += hdr->m_eff;
        S.last_err = hdr->nrm;
        if ((max_iters && cycle >= max_iters) || hdr->brokedown || hdr->nrm < tol) {
            S.breakdown = hdr->brokedown;
            break;
        }
        std::swap(ws.u[0], ws.u[krydim]);
    }
    S.passes = hdr->passes;
    S.prods = hdr->prods + 1;   // + the norm of the initial vector
    RP_CUDA(cudaMemcpyAsync(psi, ws.y, D * esize(dtype), cudaMemcpyDeviceToDevice, st));
    RP_CUDA(cudaStreamSynchronize(st));
    if (stats) *stats = S;
}

// ---------------------------------------------------------------------------
// Time-stepped primitives
// ---------------------------------------------------------------------------
void krylov_arnoldi(const ApplyPlan &plan, KryWorkspace &ws, const void *psi, int m,
                    ArnoldiResult &R, cudaStream_t st) {
    RP_REQUIRE(m >= 2 && m <= MAX_KRYLOV, -2, "m must be in [2, 64]");
    workspace_ensure(ws, plan.len, plan.dtype, m);
    const uint64_t D = ws.D;
    const int dtype = plan.dtype;
    R = ArnoldiResult{};
    R.m = m;
    R.beta0 = vec_norm(dtype, D, psi, st);
    R.H.assign((size_t)2 * m * m, 0.0);
    R.sigma.assign(m + 1, 0.0);
    if (R.beta0 == 0.0) return;
    RP_CUDA(cudaMemcpyAsync(ws.u[0], psi, D * esize(dtype), cudaMemcpyDeviceToDevice, st));
    RP_CUDA(cudaMemsetAsync(ws.err, 0, sizeof(unsigned), st));
    k_kry_init<<<1, 32, 0, st>>>(ws.dev, R.beta0);
    RP_CUDA(cudaGetLastError());
    KryDev *s = ws.dev;
    arnoldi_cycle(plan, ws, m, false, st);
    k_kry_err<<<1, 1, 0, st>>>(s, ws.err);
    RP_CUDA(cudaGetLastError());
    const KryDev &h = read_back(s, offsetof(KryDev, H) + R.H.size() * sizeof(double), st);
    std::copy(h.H, h.H + R.H.size(), R.H.begin());
    std::copy(h.sigma, h.sigma + m + 1, R.sigma.begin());
    R.m_eff = h.m_eff;
    R.breakdown = h.brokedown;
    R.passes = h.passes;
    R.beta = h.beta;
}

int krylov_lanczos(const ApplyPlan &plan, void *const *u, int m, double *alpha, double *beta, cudaStream_t st) {
    RP_REQUIRE(m >= 2 && m <= MAX_KRYLOV, -2, "m must be in [2, 64]");
    const LanczosScratch &z = lanczos_scratch();
    KryDev *s = z.dev;
    RP_CUDA(cudaMemsetAsync(z.err, 0, sizeof(unsigned), st));
    k_kry_init<<<1, 32, 0, st>>>(s, 1.0);
    k_kry_begin<<<1, 256, 0, st>>>(s, m, 0);
    RP_CUDA(cudaGetLastError());
    for (int j = 0; j < m; j++) {
        ApplyLaunch L;
        L.in = u[j];
        L.out = u[j + 1];
        L.alpha_dev = &s->sigma[j];
        L.active = &s->active;
        L.err = z.err;
        apply_launch(plan, L, st);
        lanczos_launch(plan.dtype, 1ull << plan.len, j ? u[j - 1] : nullptr, u[j], u[j + 1], s, z.partials, z.err,
                       j, j == m - 1, st);
    }
    k_kry_err<<<1, 1, 0, st>>>(s, z.err);
    RP_CUDA(cudaGetLastError());
    const KryDev &h = read_back(s, offsetof(KryDev, coef), st);
    for (int j = 0; j < h.m_eff; j++) {
        alpha[j] = h.hacc[2 * j];
        if (j < m - 1) beta[j] = h.hacc[2 * j + 1];
    }
    return h.m_eff;
}

void vec_combine(int dtype, uint64_t n, int nvec, const void *const *u, const double *coef, void *out,
                 cudaStream_t st) {
    RP_REQUIRE(nvec >= 1 && nvec <= MAX_KRYLOV, -2, "a combination takes 1 to 64 vectors");
    RP_REQUIRE(dtype == 2 || n % 2 == 0, -2, "a combination of complex64 vectors needs an even length");
    VecTable tab{};
    for (int i = 0; i < nvec; i++) tab.p[i] = u[i];
    double *c = lanczos_scratch().dev->ycoef;
    RP_CUDA(cudaMemcpyAsync(c, coef, (size_t)nvec * 2 * sizeof(double), cudaMemcpyHostToDevice, st));
    RP_CUDA(cudaMemsetAsync(out, 0, n * esize(dtype), st));
    multi_axpy(dtype, n, tab, nvec, nullptr, c, out, st);
}

void krylov_combine(KryWorkspace &ws, const ArnoldiResult &R, const double *coef, void *out,
                    cudaStream_t st) {
    RP_REQUIRE(R.m_eff >= 1 && (int)ws.u.size() >= R.m_eff, -2, "no Arnoldi basis to combine");
    std::vector<double> c((size_t)2 * R.m_eff);
    for (int i = 0; i < R.m_eff; i++) {
        c[2 * i] = coef[2 * i] * R.sigma[i];
        c[2 * i + 1] = coef[2 * i + 1] * R.sigma[i];
    }
    RP_CUDA(cudaMemcpyAsync(ws.dev->ycoef, c.data(), c.size() * sizeof(double),
                            cudaMemcpyHostToDevice, st));
    RP_CUDA(cudaMemsetAsync(out, 0, ws.D * esize(ws.dtype), st));
    VecTable tab{};
    for (int i = 0; i < R.m_eff; i++) tab.p[i] = ws.u[i];
    multi_axpy(ws.dtype, ws.D, tab, R.m_eff, nullptr, ws.dev->ycoef, out, st);
    RP_CUDA(cudaStreamSynchronize(st));
}

// One CTA per factor.  in_smem: the exponential's ten matrices fit in shared
// memory (m <= 37); in global scratch every product read back what the CTA had
// just written, past L1.  The sums are the same, bit for bit.  Measured, four
// factors, one call of rp_expm_first_columns with its copies, scratch and 256
// threads -> this: m = 16 99 -> 100 us, m = 31 250 -> 191, m = 37 321 -> 244, and by
// the threads alone m = 38 330 -> 270, m = 65 1024 -> 741.  Below m = 11 the barriers of
// 512 threads cost more than they bring (m = 4 58 us, with 256 50).
constexpr size_t CANDS_SMEM = 224 * 1024;
__global__ void __launch_bounds__(512) k_expm_cands(int m, const cd *H, const double *fr, const double *fi,
                                                    cd *scratch, cd *col0, int in_smem) {
    extern __shared__ __align__(16) unsigned char expm_smem[];
    double *fac = reinterpret_cast<double *>(expm_smem);
    const int c = blockIdx.x;
    cd *A = in_smem ? reinterpret_cast<cd *>(fac + 2 * m + 64) : scratch + (size_t)c * 10 * m * m;
    cd *E = A + (size_t)m * m, *ws = E + (size_t)m * m;
    const cd f{fr[c], fi[c]};
    for (int e = threadIdx.x; e < m * m; e += blockDim.x) A[e] = cmul(f, H[e]);
    __syncthreads();
    expm_block(m, A, E, ws, fac);
    for (int i = threadIdx.x; i < m; i += blockDim.x) col0[(size_t)c * m + i] = E[i];
}

void expm_candidates(int m, const double *H, int ncand, const double *fr, const double *fi,
                     double *col0, cudaStream_t st) {
    RP_REQUIRE(m >= 1 && m <= 1024 && ncand >= 1 && ncand <= 64, -2, "bad expm batch size");
    const size_t hb = (size_t)m * m * sizeof(cd);
    const size_t sb = (size_t)ncand * 10 * m * m * sizeof(cd);
    const size_t need = hb + sb + 2 * ncand * sizeof(double) + (size_t)ncand * m * sizeof(cd);
    // one buffer kept between calls (a step controller calls this every step)
    char *buf = static_cast<char *>(scratch_get(SCR_EXPM, need, st));
    cd *dH = (cd *)buf;
    cd *scr = (cd *)(buf + hb);
    double *dfr = (double *)(buf + hb + sb), *dfi = dfr + ncand;
    cd *dcol = (cd *)(dfi + ncand);
    RP_CUDA(cudaMemcpyAsync(dH, H, hb, cudaMemcpyHostToDevice, st));
    RP_CUDA(cudaMemcpyAsync(dfr, fr, ncand * sizeof(double), cudaMemcpyHostToDevice, st));
    RP_CUDA(cudaMemcpyAsync(dfi, fi, ncand * sizeof(double), cudaMemcpyHostToDevice, st));
    const size_t fac = (size_t)(2 * m + 64) * sizeof(double), all = fac + (size_t)10 * m * m * sizeof(cd);
    const int in_smem = all <= CANDS_SMEM;
    const size_t smem = in_smem ? all : fac;
    // the same value on every call: calls of other sizes, threads and devices cannot lower it
    RP_CUDA(cudaFuncSetAttribute(k_expm_cands, cudaFuncAttributeMaxDynamicSharedMemorySize, CANDS_SMEM));
    k_expm_cands<<<ncand, m <= 10 ? 256 : 512, smem, st>>>(m, dH, dfr, dfi, scr, dcol, in_smem);
    RP_CUDA(cudaGetLastError());
    RP_CUDA(cudaMemcpyAsync(col0, dcol, (size_t)ncand * m * sizeof(cd), cudaMemcpyDeviceToHost, st));
    RP_CUDA(cudaStreamSynchronize(st));
}

}  // namespace rp
