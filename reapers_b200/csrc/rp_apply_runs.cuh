// H.psi for small states and for term lists too long for the row kernel:
// runs of terms that share an X mask (rp_apply_runs.cu).
#pragma once

#include <cstring>
#include <vector>

#include "rp_common.cuh"

namespace rp {

// One term of a run.  c carries (-1)^popc(z & x), so the sign of output
// element n is (-1)^popc(z & n).
struct alignas(16) RunTerm {
    double c;
    uint32_t z, pad;
};

// Consecutive terms with the same X mask, nr real coefficients then ni
// imaginary ones, from term `first` on.
struct alignas(16) Run {
    uint32_t x, first, nr, ni;
};

// Host tables packed for one allocation and one copy (each at 16 bytes).
struct TablePack {
    std::vector<uint8_t> bytes;
    template <typename T>
    size_t add(const std::vector<T> &v) {
        const size_t at = bytes.size();
        bytes.resize(at + ((v.size() * sizeof(T) + 15) & ~size_t(15)), 0);
        if (!v.empty()) std::memcpy(bytes.data() + at, v.data(), v.size() * sizeof(T));
        return at;
    }
    char *upload() const {               // the tables on the device
        void *d = nullptr;
        RP_CUDA(cudaMalloc(&d, bytes.size() + 16));
        const cudaError_t e = cudaMemcpy(d, bytes.data(), bytes.size(), cudaMemcpyHostToDevice);
        if (e != cudaSuccess) cudaFree(d);
        RP_CUDA(e);
        return static_cast<char *>(d);
    }
};

struct RunPlan {
    bool ok = false;
    int eb = 0;          // log2 of the elements per lane
    int parts = 1;       // CTAs that share a block of output elements
    int nblocks = 0;     // blocks of 32 << eb output elements
    std::vector<RunTerm> terms;
    std::vector<Run> runs;               // cut at the workers' boundaries
    std::vector<uint32_t> wstart;        // worker -> first run (workers + 1 entries)
    char *dev = nullptr;                 // one allocation: terms, runs, wstart
    size_t at_runs = 0, at_wstart = 0;
};

constexpr int RUN_MIN_LEN = 5;           // smaller states: the direct kernel

// Host only: sort the terms into runs and deal them out to the workers.
void runplan_build(RunPlan &p, int len, const uint64_t *bits, const double *coeff, int64_t nterms);
void runplan_upload(RunPlan &p);
void runplan_free(RunPlan &p);
// The partial sums that all plans share (rp_shutdown).
void runs_scratch_release();

struct RunLaunch {
    const void *in = nullptr;
    void *out = nullptr;
    double alpha = 1.0;
    const double *alpha_dev = nullptr;
    int accumulate = 0;
    const int *active = nullptr;
};
void runs_launch(const RunPlan &p, int dtype, const RunLaunch &l, cudaStream_t st);

}  // namespace rp
