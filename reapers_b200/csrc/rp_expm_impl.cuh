#pragma once
// Single-CTA FP64 matrix exponential (Higham 2005, Pade 3..13 with scaling
// and squaring), included into the translation unit that launches it.
// Matrices live in global scratch (L2-resident at Krylov
// sizes); every step is a block-wide loop with __syncthreads between steps.
#include "rp_expm.cuh"

namespace rp {

// Pade numerator coefficients b_0..b_m of Higham (2005), Table 2.2.
static __constant__ double c_b13[14] = {
    64764752532480000.0, 32382376266240000.0, 7771770303897600.0, 1187353796428800.0,
    129060195264000.0,   10559470521600.0,    670442572800.0,     33522128640.0,
    1323241920.0,        40840800.0,          960960.0,           16380.0,
    182.0,               1.0};
static __constant__ double c_b9[10] = {17643225600.0, 8821612800.0, 2075673600.0, 302702400.0,
                                30270240.0,    2162160.0,    110880.0,     3960.0,
                                90.0,          1.0};
static __constant__ double c_b7[8] = {17297280.0, 8648640.0, 1995840.0, 277200.0,
                               25200.0,    1512.0,    56.0,      1.0};
static __constant__ double c_b5[6] = {30240.0, 15120.0, 3360.0, 420.0, 30.0, 1.0};
static __constant__ double c_b3[4] = {120.0, 60.0, 12.0, 1.0};

// C = A * B (n x n), block-wide.
__device__ static void mm(int n, const cd *A, const cd *B, cd *C) {
    const int nn = n * n;
    for (int e = threadIdx.x; e < nn; e += blockDim.x) {
        const int i = e % n, j = e / n;
        double sr = 0.0, si = 0.0;
        for (int k = 0; k < n; k++) {
            const cd a = A[i + k * n], b = B[k + j * n];
            sr = fma(a.x, b.x, fma(-a.y, b.y, sr));
            si = fma(a.x, b.y, fma(a.y, b.x, si));
        }
        C[e] = cd{sr, si};
    }
    __syncthreads();
}

// Solve Q X = P in place (X -> P), Gaussian elimination with partial pivoting.
__device__ static void solve(int n, cd *Q, cd *P, double *smem) {
    double *fac = smem;              // 2n doubles: elimination factors
    __shared__ int s_piv;
    __shared__ double s_best[32];
    __shared__ int s_idx[32];
    for (int k = 0; k < n; k++) {
        // pivot search over rows k..n-1 of column k
        double best = -1.0;
        int bi = k;
        for (int i = k + threadIdx.x; i < n; i += blockDim.x) {
            const cd q = Q[i + k * n];
            const double v = hypot(q.x, q.y);
            if (v > best) { best = v; bi = i; }
        }
        for (int o = 16; o > 0; o >>= 1) {
            const double ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int oi = __shfl_xor_sync(0xffffffffu, bi, o);
            if (ob > best || (ob == best && oi < bi)) { best = ob; bi = oi; }
        }
        if ((threadIdx.x & 31) == 0) { s_best[threadIdx.x >> 5] = best; s_idx[threadIdx.x >> 5] = bi; }
        __syncthreads();
        if (threadIdx.x == 0) {
            double b = -1.0;
            int p = k;
            for (int w = 0; w < (int)(blockDim.x >> 5); w++)
                if (s_best[w] > b || (s_best[w] == b && s_idx[w] < p)) { b = s_best[w]; p = s_idx[w]; }
            s_piv = p;
        }
        __syncthreads();
        const int p = s_piv;
        if (p != k) {
            for (int j = threadIdx.x; j < n; j += blockDim.x) {
                cd t = Q[k + j * n]; Q[k + j * n] = Q[p + j * n]; Q[p + j * n] = t;
                t = P[k + j * n]; P[k + j * n] = P[p + j * n]; P[p + j * n] = t;
            }
        }
        __syncthreads();
        const cd d = Q[k + k * n];
        for (int i = k + 1 + threadIdx.x; i < n; i += blockDim.x) {
            const cd f = cdiv(Q[i + k * n], d);
            fac[2 * i] = f.x;
            fac[2 * i + 1] = f.y;
        }
        __syncthreads();
        const int rows = n - k - 1;
        for (int e = threadIdx.x; e < rows * 2 * n; e += blockDim.x) {
            const int i = k + 1 + e % rows;
            const int jj = e / rows;   // 0..2n-1: columns of Q then of P
            const cd f{fac[2 * i], fac[2 * i + 1]};
            if (jj < n) {
                if (jj >= k) {
                    const cd a = Q[k + jj * n], t = cmul(f, a);
                    Q[i + jj * n].x -= t.x;
                    Q[i + jj * n].y -= t.y;
                }
            } else {
                const int j = jj - n;
                const cd a = P[k + j * n], t = cmul(f, a);
                P[i + j * n].x -= t.x;
                P[i + j * n].y -= t.y;
            }
        }
        __syncthreads();
    }
    // back substitution, one column of P per thread group
    for (int i = n - 1; i >= 0; i--) {
        const cd d = Q[i + i * n];
        for (int j = threadIdx.x; j < n; j += blockDim.x) {
            double sr = P[i + j * n].x, si = P[i + j * n].y;
            for (int k = i + 1; k < n; k++) {
                const cd q = Q[i + k * n], x = P[k + j * n];
                sr -= q.x * x.x - q.y * x.y;
                si -= q.x * x.y + q.y * x.x;
            }
            P[i + j * n] = cdiv(cd{sr, si}, d);
        }
        __syncthreads();
    }
}

__device__ inline void expm_block(int n, const cd *A_in, cd *E, cd *scratch, double *smem) {
    const int nn = n * n;
    cd *A = scratch, *A2 = A + nn, *A4 = A2 + nn, *A6 = A4 + nn;
    cd *U = A6 + nn, *V = U + nn, *T = V + nn, *Pm = T + nn;
    __shared__ double s_norm;
    __shared__ double s_colmax[32];
    // 1-norm (max column sum of |a_ij|)
    double best = 0.0;
    for (int j = threadIdx.x; j < n; j += blockDim.x) {
        double s = 0.0;
        for (int i = 0; i < n; i++) s += hypot(A_in[i + j * n].x, A_in[i + j * n].y);
        best = fmax(best, s);
    }
    for (int o = 16; o > 0; o >>= 1) best = fmax(best, __shfl_xor_sync(0xffffffffu, best, o));
    if ((threadIdx.x & 31) == 0) s_colmax[threadIdx.x >> 5] = best;
    __syncthreads();
    if (threadIdx.x == 0) {
        double b = 0.0;
        for (int w = 0; w < (int)(blockDim.x >> 5); w++) b = fmax(b, s_colmax[w]);
        s_norm = b;
    }
    __syncthreads();
    const double a1 = s_norm;
    int deg, s = 0;
    if (a1 <= 1.495585217958292e-2) deg = 3;
    else if (a1 <= 2.539398330063230e-1) deg = 5;
    else if (a1 <= 9.504178996162932e-1) deg = 7;
    else if (a1 <= 2.097847961257068e0) deg = 9;
    else {
        deg = 13;
        const double r = a1 / 5.371920351148152e0;
        if (r > 1.0) s = (int)ceil(log2(r));
    }
    const double sc = ldexp(1.0, -s);
    for (int e = threadIdx.x; e < nn; e += blockDim.x) A[e] = cd{A_in[e].x * sc, A_in[e].y * sc};
    __syncthreads();
    mm(n, A, A, A2);
    if (deg == 13) {
        mm(n, A2, A2, A4);
        mm(n, A4, A2, A6);
        for (int e = threadIdx.x; e < nn; e += blockDim.x) {
            T[e] = cd{c_b13[13] * A6[e].x + c_b13[11] * A4[e].x + c_b13[9] * A2[e].x,
                      c_b13[13] * A6[e].y + c_b13[11] * A4[e].y + c_b13[9] * A2[e].y};
        }
        __syncthreads();
        mm(n, A6, T, Pm);
        for (int e = threadIdx.x; e < nn; e += blockDim.x) {
            const int i = e % n, j = e / n;
            cd p = Pm[e];
            p.x += c_b13[7] * A6[e].x + c_b13[5] * A4[e].x + c_b13[3] * A2[e].x + (i == j ? c_b13[1] : 0.0);
            p.y += c_b13[7] * A6[e].y + c_b13[5] * A4[e].y + c_b13[3] * A2[e].y;
            Pm[e] = p;
            T[e] = cd{c_b13[12] * A6[e].x + c_b13[10] * A4[e].x + c_b13[8] * A2[e].x,
                      c_b13[12] * A6[e].y + c_b13[10] * A4[e].y + c_b13[8] * A2[e].y};
        }
        __syncthreads();
        mm(n, A, Pm, U);
        mm(n, A6, T, V);
        for (int e = threadIdx.x; e < nn; e += blockDim.x) {
            const int i = e % n, j = e / n;
            cd v = V[e];
            v.x += c_b13[6] * A6[e].x + c_b13[4] * A4[e].x + c_b13[2] * A2[e].x + (i == j ? c_b13[0] : 0.0);
            v.y += c_b13[6] * A6[e].y + c_b13[4] * A4[e].y + c_b13[2] * A2[e].y;
            V[e] = v;
        }
        __syncthreads();
    } else {
        const double *b = deg == 3 ? c_b3 : deg == 5 ? c_b5 : deg == 7 ? c_b7 : c_b9;
        // Pm = A^(2k), accumulated into V (even part) and T (odd part / A)
        for (int e = threadIdx.x; e < nn; e += blockDim.x) {
            const int i = e % n, j = e / n;
            const double id = i == j ? 1.0 : 0.0;
            Pm[e] = cd{id, 0.0};
            V[e] = cd{b[0] * id, 0.0};
            T[e] = cd{b[1] * id, 0.0};
        }
        __syncthreads();
        for (int k = 1; 2 * k <= deg; k++) {
            mm(n, Pm, A2, A4);   // A4 as the next power
            for (int e = threadIdx.x; e < nn; e += blockDim.x) {
                const cd p = A4[e];
                Pm[e] = p;
                V[e].x += b[2 * k] * p.x;
                V[e].y += b[2 * k] * p.y;
                T[e].x += b[2 * k + 1] * p.x;
                T[e].y += b[2 * k + 1] * p.y;
            }
            __syncthreads();
        }
        mm(n, A, T, U);
    }
    // (V - U) X = (V + U)
    for (int e = threadIdx.x; e < nn; e += blockDim.x) {
        const cd u = U[e], v = V[e];
        T[e] = cd{v.x - u.x, v.y - u.y};
        Pm[e] = cd{v.x + u.x, v.y + u.y};
    }
    __syncthreads();
    solve(n, T, Pm, smem);
    for (int k = 0; k < s; k++) {
        mm(n, Pm, Pm, T);
        for (int e = threadIdx.x; e < nn; e += blockDim.x) Pm[e] = T[e];
        __syncthreads();
    }
    for (int e = threadIdx.x; e < nn; e += blockDim.x) E[e] = Pm[e];
    __syncthreads();
}

// ---------------------------------------------------------------------------
// First column of exp(f H) by the truncated Taylor series on s equal pieces of
// the factor: y <- sum_{k <= K} (f H / s)^k y / k!, s times from e_1.
//
// The Krylov methods use column 0 alone, and Hfull is block lower bidiagonal
// (diagonal blocks of the cycles' Hessenberg matrices, one coupling entry
// between neighbours), so a term is a product with nblk m^2 entries, where the
// Pade form multiplies and solves with n^2 matrices.  f H is shifted by the mean
// of its diagonal (the factor e^mu comes back at the end); a piece has 1-norm at
// most 2, K is the smallest with theta^K / K! below 2^-55 of it.  Rounding errors
// add up over the pieces like over Pade's squarings: against extended precision
// both are at 1e-16 to 3e-15 for norms up to 100 (random Hessenberg matrices,
// real, imaginary and complex f).
//
// One CTA, eight threads per row, one barrier per term: bound by the latency of
// that chain (0.4 us).  Measured, us per exponential of an evolve, Pade -> this:
// n = 16, 32, 48 (17 qubits, t = 5) 287 -> 59 on average; n = 20, 40 (dense SYK)
// 238 -> 28; n = 24, 48, 72, 96 (20-qubit chain) 1314 -> 244.
// ---------------------------------------------------------------------------
constexpr int ACT_T = 8;                 // threads per row
constexpr int ACT_Q = 8;                 // entries of a row a thread can hold
constexpr int ACT_KMAX = 40;
// Measured cost in us: a term with a row per group (its entries in registers),
// a term otherwise, per round of rows (constant and per entry), and Pade-13 with
// its squarings (constant and per n^3).  Large norms, and with them hundreds of
// pieces, go to Pade.
constexpr double ACT_TERM_US = 0.4, ACT_ROUND_US = 0.35, ACT_ENTRY_US = 0.07, PADE_US = 100.0,
                 PADE_N3_US = 3.7e-3;
// Largest exponent by which the sum may grow on its way, and the largest of e^(mu/2)
// (a double ends at e^709): the shifted sum grows like e^(norm of its Hermitian
// part) although exp(f H) itself may stay below one.  Beyond it: Pade, which
// scales the matrix as a whole.
constexpr double ACT_MAX_EXP = 600.0;

// H as its blocks: block b (rows and columns b m ..., the last of order mlast)
// at blk + b * stride (row-major, leading dimension m), coupling entry sub[b] at
// (b m, b m - 1) for b > 0.  All of it is rewritten (scaled and shifted).
// hess: the blocks are upper Hessenberg (nothing is read below).
struct ActionMatrix {
    cd *blk;
    cd *sub;
    int m, nblk, mlast;
    bool hess;
};

// v, w, y: n entries each in shared memory.  True: y = column 0 of exp(f H);
// false: too many pieces, or sums beyond a double's range; the caller takes Pade
// (blk is left scaled by f).
__device__ inline bool expm_action(const ActionMatrix a, cd f, cd *v, cd *w, cd *y) {
    __shared__ double s_col[32];
    __shared__ cd s_mu;
    __shared__ int s_pieces, s_terms;
    __shared__ double s_rk[ACT_KMAX];
    const int n = (a.nblk - 1) * a.m + a.mlast, m = a.m;
    const int tid = threadIdx.x, lane = tid & 31, warp = tid >> 5, nw = blockDim.x >> 5;
    // A = f H, and the mean of its diagonal
    for (int e = tid; e < a.nblk * m * m; e += blockDim.x) a.blk[e] = cmul(f, a.blk[e]);
    for (int b = tid; b < a.nblk; b += blockDim.x) a.sub[b] = b ? cmul(f, a.sub[b]) : cd{0.0, 0.0};
    __syncthreads();
    if (warp == 0) {
        double tr = 0.0, ti = 0.0;
        for (int i = lane; i < n; i += 32) {
            const cd d = a.blk[(size_t)(i / m) * m * m + (size_t)(i % m) * (m + 1)];
            tr += d.x;
            ti += d.y;
        }
        tr = warp_sum(tr);
        ti = warp_sum(ti);
        if (lane == 0) s_mu = cd{tr / n, ti / n};
    }
    __syncthreads();
    const cd mu = s_mu;
    // 1-norm of A - mu (HERM: of its Hermitian part), a warp per column
    auto norm1 = [&](bool herm) {
        double best = 0.0;
        for (int j = warp; j < n; j += nw) {
            const int b = j / m, c = j % m, rows = b == a.nblk - 1 ? a.mlast : m;
            const cd *const blk = a.blk + (size_t)b * m * m;
            double s = 0.0;
            for (int i = lane; i < rows; i += 32) {
                cd q = blk[(size_t)i * m + c];
                if (i == c) q = cd{q.x - mu.x, q.y - mu.y};
                if (herm) {
                    cd p = blk[(size_t)c * m + i];
                    if (i == c) p = cd{p.x - mu.x, p.y - mu.y};
                    q = cd{0.5 * (q.x + p.x), 0.5 * (q.y - p.y)};
                }
                s += sqrt(q.x * q.x + q.y * q.y);
            }
            auto coupling = [&](int k) {
                const cd q = a.sub[k];
                s += (herm ? 0.5 : 1.0) * sqrt(q.x * q.x + q.y * q.y);
            };
            if (lane == 0 && c == m - 1 && b + 1 < a.nblk) coupling(b + 1);
            if (lane == 0 && herm && c == 0 && b > 0) coupling(b);
            s = warp_sum(s);
            // (a NaN stays: fmax would drop it)
            best = s > best || s != s ? s : best;
        }
        __syncthreads();
        if (lane == 0) s_col[warp] = best;
        __syncthreads();
        double nrm = 0.0;
        for (int i = 0; i < nw; i++) nrm = s_col[i] > nrm || s_col[i] != s_col[i] ? s_col[i] : nrm;
        return nrm;                      // the same in every thread
    };
    const double nrm = norm1(false);
    if (!(nrm < 1e6)) return false;      // (an infinite or NaN norm too)
    if (nrm > ACT_MAX_EXP && !(norm1(true) <= ACT_MAX_EXP)) return false;
    if (fabs(mu.x) > 2.0 * ACT_MAX_EXP) return false;
    if (tid == 0) {
        const int pieces = nrm > 2.0 ? (int)ceil(0.5 * nrm) : 1;
        const double theta = nrm / pieces;
        int terms = 1;
        for (double t = theta; t > 2.8e-17 && terms < ACT_KMAX;) t *= theta / ++terms;
        const int groups = (int)blockDim.x / ACT_T, entries = (m + ACT_T - 1) / ACT_T;
        const double term = n <= groups && entries <= ACT_Q
                                ? ACT_TERM_US
                                : (n + groups - 1) / groups * (ACT_ROUND_US + ACT_ENTRY_US * entries);
        const double n3 = (double)n * n * n;
        s_pieces = term * pieces * terms <= PADE_US + PADE_N3_US * n3 ? pieces : 0;
        s_terms = terms;
    }
    __syncthreads();
    const int pieces = s_pieces, terms = s_terms;
    if (pieces == 0) return false;
    const double inv = 1.0 / pieces;
    for (int e = tid; e < a.nblk * m * m; e += blockDim.x) {
        cd q = a.blk[e];
        const int i = (e % (m * m)) / m, j = e % m;
        if (i == j) q = cd{q.x - mu.x, q.y - mu.y};
        a.blk[e] = cd{q.x * inv, q.y * inv};
    }
    for (int b = tid; b < a.nblk; b += blockDim.x) a.sub[b] = cd{a.sub[b].x * inv, a.sub[b].y * inv};
    for (int i = tid; i < n; i += blockDim.x) v[i] = y[i] = cd{i == 0 ? 1.0 : 0.0, 0.0};
    __syncthreads();
    for (int k = tid; k < ACT_KMAX; k += blockDim.x) s_rk[k] = 1.0 / (k + 1);
    __syncthreads();
    const int t = tid % ACT_T, group = tid / ACT_T, groups = blockDim.x / ACT_T;
    if (n <= groups && m <= ACT_T * ACT_Q) {
        // one row per group: its entries stay in registers
        const bool own = group < n;
        const int b = own ? group / m : 0, r = own ? group - b * m : 0;
        const int cols = !own ? 0 : b == a.nblk - 1 ? a.mlast : m;
        const cd *row = a.blk + ((size_t)b * m + r) * m;
        cd q[ACT_Q];
#pragma unroll
        for (int c = 0; c < ACT_Q; c++) q[c] = t + ACT_T * c < cols ? row[t + ACT_T * c] : cd{0.0, 0.0};
        const cd link = own && t == 0 && r == 0 && b ? a.sub[b] : cd{0.0, 0.0};
        const bool linked = own && t == 0 && r == 0 && b;
        const int nq = (m + ACT_T - 1) / ACT_T;
        cd sum = own ? y[group] : cd{0.0, 0.0};
        // the warps that have rows, behind a barrier of their own
        const int busy = (n * ACT_T + 31) & ~31;
        for (int s = 0; s < pieces && tid < busy; s++) {
            for (int k = 0; k < terms; k++) {
                const cd *x = v + b * m + t;
                double rr = 0.0, ri = 0.0, ir = 0.0, ii = 0.0;
#pragma unroll
                for (int c = 0; c < ACT_Q; c++) {
                    if (c < nq) {
                        const cd z = x[t + ACT_T * c < cols ? ACT_T * c : -t];
                        rr = fma(q[c].x, z.x, rr);
                        ii = fma(q[c].y, z.y, ii);
                        ri = fma(q[c].x, z.y, ri);
                        ir = fma(q[c].y, z.x, ir);
                    }
                }
                if (linked) {
                    const cd z = v[group - 1];
                    rr = fma(link.x, z.x, rr);
                    ii = fma(link.y, z.y, ii);
                    ri = fma(link.x, z.y, ri);
                    ir = fma(link.y, z.x, ir);
                }
                double sr = rr - ii, si = ri + ir;
#pragma unroll
                for (int o = ACT_T / 2; o > 0; o >>= 1) {
                    sr += __shfl_xor_sync(0xffffffffu, sr, o);
                    si += __shfl_xor_sync(0xffffffffu, si, o);
                }
                const cd term{sr * s_rk[k], si * s_rk[k]};
                sum.x += term.x;
                sum.y += term.y;
                if (own && t == 0) w[group] = k == terms - 1 ? sum : term;   // the next piece starts from the sum
                asm volatile("bar.sync 1, %0;" ::"r"(busy) : "memory");
                cd *const z = v;
                v = w;
                w = z;
            }
        }
        if (own && t == 0) y[group] = sum;
        __syncthreads();
    } else {
        for (int s = 0; s < pieces; s++) {
            for (int k = 0; k < terms; k++) {
                const double rk = s_rk[k];
                for (int i = group; i < n; i += groups) {
                    const int b = i / m, r = i - b * m, cols = b == a.nblk - 1 ? a.mlast : m;
                    const cd *row = a.blk + ((size_t)b * m + r) * m;
                    const cd *x = v + b * m;
                    double sr = 0.0, si = 0.0;
                    const int j0 = a.hess && r > 0 ? (r - 1) & ~(ACT_T - 1) : 0;
#pragma unroll 4
                    for (int j = j0 + t; j < cols; j += ACT_T) {
                        const cd q = row[j], z = x[j];
                        sr = fma(q.x, z.x, fma(-q.y, z.y, sr));
                        si = fma(q.x, z.y, fma(q.y, z.x, si));
                    }
                    if (t == 0 && r == 0 && b) {
                        const cd q = a.sub[b], z = v[i - 1];
                        sr = fma(q.x, z.x, fma(-q.y, z.y, sr));
                        si = fma(q.x, z.y, fma(q.y, z.x, si));
                    }
                    // the groups of a warp may differ in their last row:
                    // shuffle among the eight threads of this one
                    const unsigned mask = 0xffu << (lane & ~(ACT_T - 1));
#pragma unroll
                    for (int o = ACT_T / 2; o > 0; o >>= 1) {
                        sr += __shfl_xor_sync(mask, sr, o);
                        si += __shfl_xor_sync(mask, si, o);
                    }
                    if (t == 0) {
                        const cd q{sr * rk, si * rk};
                        const cd sum{y[i].x + q.x, y[i].y + q.y};
                        y[i] = sum;
                        w[i] = k == terms - 1 ? sum : q;
                    }
                }
                __syncthreads();
                cd *const z = v;
                v = w;
                w = z;
            }
        }
    }
    // e^mu in two halves: y may be as large as e^mu is small
    const double er = exp(0.5 * mu.x);
    double sn, cs;
    sincos(mu.y, &sn, &cs);
    for (int i = tid; i < n; i += blockDim.x) {
        const cd q = cmul(cd{er * cs, er * sn}, y[i]);
        y[i] = cd{er * q.x, er * q.y};
    }
    __syncthreads();
    return true;
}

}  // namespace rp
