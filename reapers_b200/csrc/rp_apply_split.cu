// Split row kernel: the row layout of rp_apply_rows.cu (256-row tiles of 128
// bytes brought in by swizzled TMA copies, consumer thread = output row) for
// states of 2^5 or 2^6 such tiles, where one CTA per tile would leave most of
// the GPU idle.  A cluster of C CTAs computes an output tile: each streams the
// source tiles of its share of the terms, then the C partial tiles meet
// through distributed shared memory, CTA r adding rows [r 256/C, (r+1) 256/C)
// over the ranks in order (results are the same run to run) and writing them.
// Bound by the shared-memory gathers (8 or 16 bytes per element and term at
// 128 B/clk/SM) and the cluster's two barriers.  Sparse SYK: 2^17 complex64,
// 272 terms 106 -> 21.2 us (gathers alone 7.8 us), 2^18, 288 terms 132 -> 33
// us (16.6 us), against the tiled kernel's one CTA per 2^9- or 2^10-element
// tile.
#include <cooperative_groups.h>
#include <cuda.h>

#include <algorithm>

#include "rp_apply.cuh"
#include "rp_apply_split.cuh"
#include "rp_rows_dev.cuh"

namespace cg = cooperative_groups;

namespace rp {

template <typename Real>
struct SplitArgs {
    Cplx<Real> *out;
    const SplitPart *part;
    const RowTerm<float> *terms;
    const RowGroup *groups;
    const RowDiag *diag;
    const uint32_t *dstart;
    int parts, stages, max_terms, max_groups, ndiag;
    double alpha;
    const double *alpha_dev;
    int accumulate;
    const int *active;
    unsigned *err;
};

template <typename Real, bool DIAG>
__global__ void __launch_bounds__(ROW_P + 32, 2)
    k_apply_split(const __grid_constant__ CUtensorMap tmap, const SplitArgs<Real> a) {
    constexpr int C = 128 / (int)sizeof(Cplx<Real>);   // elements per row
    constexpr int LOGC = C == 16 ? 4 : 3;
    constexpr int B = LOGC + 8;
    extern __shared__ unsigned char smem_raw[];
    // 1024-byte alignment for the 128-byte swizzle pattern
    unsigned char *stage = reinterpret_cast<unsigned char *>(
        (reinterpret_cast<uintptr_t>(smem_raw) + 1023) & ~uintptr_t(1023));
    const int S = a.stages;
    RowTerm<float> *sterms = reinterpret_cast<RowTerm<float> *>(stage + (size_t)S * ROW_TILE_BYTES);
    RowGroup *sgroups = reinterpret_cast<RowGroup *>(sterms + a.max_terms);
    RowDiag *sdiag = reinterpret_cast<RowDiag *>(sgroups + a.max_groups);
    uint32_t *sdstart = reinterpret_cast<uint32_t *>(sdiag + (DIAG ? a.ndiag : 0));
    uint64_t *full = reinterpret_cast<uint64_t *>(sdstart + (DIAG ? (C + 4) & ~3 : 0));
    uint64_t *empty = full + S;
    __shared__ int s_abort;
    __shared__ int s_issued;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned rank = blockIdx.x % (unsigned)a.parts;
    const uint32_t o = blockIdx.x / (unsigned)a.parts;   // output tile
    const SplitPart pt = a.part[rank];
    for (int i = tid; i < (int)pt.nt; i += blockDim.x) sterms[i] = a.terms[pt.t0 + i];
    for (int i = tid; i < (int)pt.ng; i += blockDim.x) sgroups[i] = a.groups[pt.g0 + i];
    if constexpr (DIAG) {
        if (pt.diag) {
            for (int i = tid; i < a.ndiag; i += blockDim.x) sdiag[i] = a.diag[i];
            for (int i = tid; i <= C; i += blockDim.x) sdstart[i] = a.dstart[i];
        }
    }
    if (tid == 0) {
        for (int s = 0; s < S; s++) {
            mbar_init(&full[s], 1);
            mbar_init(&empty[s], ROW_NW);
        }
        s_abort = 0;
        s_issued = 0;
        fence_barrier_init();
    }
    wait_prior_kernel();
    if (a.active && *a.active == 0) return;   // the same in every CTA of the cluster
    __syncthreads();

    Cplx<Real> acc[C];
#pragma unroll
    for (int u = 0; u < C; u++) acc[u].x = acc[u].y = Real(0);
    const int ng = (int)pt.ng;
    if (warp == ROW_NW) {
        if (lane == 0) {
            asm volatile("prefetch.tensormap [%0];" ::"l"(reinterpret_cast<uint64_t>(&tmap)) : "memory");
            int g = 0;
            for (; g < ng; ++g) {
                const int s = g % S;
                if (!mbar_wait_bounded(&empty[s], (unsigned)((g / S) & 1) ^ 1u, a.err)) {
                    atomicExch(&s_abort, 1);
                    break;
                }
                mbar_arrive_expect_tx(&full[s], ROW_TILE_BYTES);
                tma_load_2d(stage + (size_t)s * ROW_TILE_BYTES, &tmap, 0,
                            (int)((o ^ sgroups[g].xh) * 256u), &full[s]);
            }
            s_issued = g;
        }
    } else {
        const uint32_t row = (uint32_t)tid;
        for (int g = 0; g < ng; ++g) {
            const int s = g % S;
            const RowGroup gd = sgroups[g];
            const uint32_t src_hi = (o ^ gd.xh) << B;
            if (!mbar_wait_bounded(&full[s], (unsigned)((g / S) & 1), a.err)) {
                atomicExch(&s_abort, 1);
                break;
            }
            const uint32_t tile = smem_u32(stage + (size_t)s * ROW_TILE_BYTES);
            apply_group<Real, DIAG ? 1 : 0>(acc, sterms, gd.first, gd.first + gd.count, src_hi, row, tile);
            if constexpr (DIAG) {
                if (g == 0 && pt.diag)
                    apply_diag<Real, false>(acc, sdiag, sdstart, (o << 8) | row,
                                            (tile + row * 128u) | ((row & 7u) << 4), 0u);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[s]);
        }
    }
    __syncthreads();
    if (s_abort && tid == 0) {
        // let the copies still in flight land before the stages are reused
        for (int g = std::max(0, s_issued - S); g < s_issued; ++g)
            mbar_wait_bounded(&full[g % S], (unsigned)((g / S) & 1), a.err);
    }
    __syncthreads();
    // the partial tile into stage 0 (chunk p of row r at chunk p ^ (r & 7));
    // after an abort it is incomplete, and the error word says so
    float4 *mine = reinterpret_cast<float4 *>(stage);
    if (tid < ROW_P) {
#pragma unroll
        for (int p = 0; p < 8; p++) mine[tid * 8 + (p ^ (tid & 7))] = row_chunk<Real>(acc, p);
    }
    cg::cluster_group cl = cg::this_cluster();
    cl.sync();
    const double scale = a.alpha * (a.alpha_dev ? *a.alpha_dev : 1.0);
    const int per = 2048 / a.parts;      // 16-byte chunks of this CTA's rows
    for (int i = tid; i < per; i += blockDim.x) {
        const int ch = (int)rank * per + i, row = ch >> 3, p = ch & 7;
        const int at = row * 8 + (p ^ (row & 7));
        constexpr int EPC = 16 / (int)sizeof(Cplx<Real>);
        Cplx<Real> s[EPC];
        *reinterpret_cast<float4 *>(s) = *cl.map_shared_rank(mine + at, 0);
        for (int c = 1; c < a.parts; c++) {
            Cplx<Real> q[EPC];
            *reinterpret_cast<float4 *>(q) = *cl.map_shared_rank(mine + at, c);
#pragma unroll
            for (int e = 0; e < EPC; e++) {
                s[e].x += q[e].x;
                s[e].y += q[e].y;
            }
        }
        float4 *dst = reinterpret_cast<float4 *>(a.out + ((size_t)o << B)) + ch;
        if (a.accumulate) {
            Cplx<Real> old[EPC];
            *reinterpret_cast<float4 *>(old) = *dst;
#pragma unroll
            for (int e = 0; e < EPC; e++) {
                s[e].x = (Real)(scale * (double)s[e].x) + old[e].x;
                s[e].y = (Real)(scale * (double)s[e].y) + old[e].y;
            }
        } else {
#pragma unroll
            for (int e = 0; e < EPC; e++) {
                s[e].x = (Real)(scale * (double)s[e].x);
                s[e].y = (Real)(scale * (double)s[e].y);
            }
        }
        *dst = *reinterpret_cast<float4 *>(s);
    }
    cl.sync();   // no CTA leaves while another reads its tile
}

// ---------------------------------------------------------------------------
// Host
// ---------------------------------------------------------------------------

// Shared-memory traffic in row loads: a term reads the row once, a source tile
// is written once; the fused diagonal reads it once and sums its terms.
static double group_cost(const RowPlan &rp, const RowGroup &g, size_t gi) {
    return 1.0 + g.count + (rp.ndiag && gi == 0 ? 1.0 + 0.15 * rp.ndiag : 0.0);
}

void splitplan_cut(SplitPlan &p, int parts) {
    const RowPlan &rp = p.rows;
    p.parts = parts;
    p.part.clear();
    p.groups.clear();
    p.terms = rp.terms;
    double total = 0.0;
    for (size_t g = 0; g < rp.groups.size(); g++) total += group_cost(rp, rp.groups[g], g);
    double load = 0.0, rest = total;   // this part's so far; what is not dealt out
    p.part.push_back({0u, 0u, 0u, 0u, rp.ndiag ? 1u : 0u});
    auto full_share = [&](double next) {
        const int left = parts - (int)p.part.size() + 1;   // this part and those after
        return left > 1 && load > 0.0 && load + 0.5 * next >= (load + rest) / left;
    };
    auto next_part = [&](uint32_t t) {
        load = 0.0;
        p.part.push_back({(uint32_t)p.groups.size(), 0u, t, 0u, 0u});
    };
    auto open = [&](uint32_t xh, uint32_t t) {
        p.groups.push_back({xh, t - p.part.back().t0, 0u, 0u});
        p.part.back().ng++;
    };
    for (size_t g = 0; g < rp.groups.size(); g++) {
        const RowGroup &gd = rp.groups[g];
        const double head = group_cost(rp, gd, g) - gd.count;
        if (full_share(head + 1.0)) next_part(gd.first);
        open(gd.xh, gd.first);
        load += head;
        rest -= head;
        for (uint32_t t = gd.first; t < gd.first + gd.count; t++) {
            if (t > gd.first && full_share(1.0)) {
                // the group goes on in the next part, which loads its tile again
                next_part(t);
                open(gd.xh, t);
                load += 1.0;
                p.terms[t].cs &= ~ROW_SAME_SRC;
            }
            p.groups.back().count++;
            p.part.back().nt++;
            load += 1.0;
            rest -= 1.0;
        }
    }
    while ((int)p.part.size() < parts)
        p.part.push_back({(uint32_t)p.groups.size(), 0u, (uint32_t)p.terms.size(), 0u, 0u});
    p.max_terms = p.max_groups = 0;
    for (const SplitPart &s : p.part) {
        p.max_terms = std::max(p.max_terms, (int)s.nt);
        p.max_groups = std::max(p.max_groups, (int)s.ng);
    }
}

// Shared memory of a launch beside its stages: a part's tables, the diagonal, and
// the slack of the swizzle's alignment.
static size_t split_fixed_bytes(const SplitPlan &p) {
    return (size_t)p.max_terms * sizeof(RowTerm<float>) + (size_t)p.max_groups * sizeof(RowGroup) +
           (p.rows.ndiag ? (size_t)p.rows.ndiag * sizeof(RowDiag) + (size_t)(((1 << p.rows.logC) + 4) & ~3) * 4 : 0) +
           1024;
}

// Stages that fit beside them with two CTAs per SM, 3 at most; one will do.
static int split_stages(size_t fixed) {
    const size_t budget = 113 * 1024 - 64 - 16 * 8;
    return fixed < budget ? (int)std::min<size_t>(3, (budget - fixed) / (ROW_TILE_BYTES + 16)) : 0;
}

void splitplan_build(SplitPlan &p, int len, int dtype, const uint64_t *bits, const double *coeff,
                     int64_t nterms) {
    p = SplitPlan{};
    rowplan_build(p.rows, len, dtype, bits, coeff, nterms, true, true);
    // (from 128 tiles on a list without a row plan is too long for this kernel too)
    if (!p.rows.ok || p.rows.groups.empty() || p.rows.ntiles >= 128) return;
    // as many CTAs per tile as fit on the GPU at once, two per SM
    int parts = 1;
    while (parts < 8 && p.rows.ntiles * parts * 2 <= 2 * num_sms()) parts *= 2;
    splitplan_cut(p, parts);
    p.ok = split_stages(split_fixed_bytes(p)) >= 1;
}

void splitplan_upload(SplitPlan &p) {
    if (!p.ok) return;
    splitplan_free(p);
    TablePack t;
    t.add(p.terms);
    p.at_groups = t.add(p.groups);
    p.at_part = t.add(p.part);
    p.at_diag = t.add(p.rows.diag);
    p.at_dstart = t.add(p.rows.dstart);
    p.dev = t.upload();
}

void splitplan_free(SplitPlan &p) {
    if (p.dev) cudaFree(p.dev);
    p.dev = nullptr;
}

template <typename Real, bool DIAG>
static void launch_split(const SplitPlan &p, int len, int dtype, const RowLaunch &l, cudaStream_t st) {
    const size_t fixed = split_fixed_bytes(p);
    const int S = split_stages(fixed);
    RP_REQUIRE(S >= 1, -2, "Hamiltonian table too large for the split row kernel");
    const size_t smem = (size_t)S * ROW_TILE_BYTES + fixed + (size_t)2 * S * sizeof(uint64_t);
    auto kern = k_apply_split<Real, DIAG>;
    static size_t attr_smem = 0;
    if (smem > attr_smem) {
        RP_CUDA(cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
        attr_smem = smem;
    }
    SplitArgs<Real> a;
    a.out = static_cast<Cplx<Real> *>(l.out);
    a.part = reinterpret_cast<const SplitPart *>(p.dev + p.at_part);
    a.terms = reinterpret_cast<const RowTerm<float> *>(p.dev);
    a.groups = reinterpret_cast<const RowGroup *>(p.dev + p.at_groups);
    a.diag = reinterpret_cast<const RowDiag *>(p.dev + p.at_diag);
    a.dstart = reinterpret_cast<const uint32_t *>(p.dev + p.at_dstart);
    a.parts = p.parts;
    a.stages = S;
    a.max_terms = p.max_terms;
    a.max_groups = p.max_groups;
    a.ndiag = p.rows.ndiag;
    a.alpha = l.alpha;
    a.alpha_dev = l.alpha_dev;
    a.accumulate = l.accumulate;
    a.active = l.active;
    a.err = l.err;
    const CUtensorMap map = make_row_map(l.in, len, dtype);
    launch_dependent(kern, p.rows.ntiles * p.parts, ROW_P + 32, smem, st, p.parts, map, a);
}

void split_launch(const SplitPlan &p, int len, int dtype, const RowLaunch &l, cudaStream_t st) {
    RP_REQUIRE(p.ok, -2, "split row kernel not planned for this Hamiltonian");
    if (dtype == 2) {
        if (p.rows.ndiag) launch_split<double, true>(p, len, dtype, l, st);
        else launch_split<double, false>(p, len, dtype, l, st);
    } else {
        if (p.rows.ndiag) launch_split<float, true>(p, len, dtype, l, st);
        else launch_split<float, false>(p, len, dtype, l, st);
    }
}

}  // namespace rp
