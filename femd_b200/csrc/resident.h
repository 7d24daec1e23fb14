// resident.h -- the on-chip Jacobi-PCG of resident.cu, for the solve entry points of krylov.cu.
#pragma once

#include "common.cuh"

namespace femd {

// What the kernel leaves for the host.
struct ResidentOut {
    double nb, rn, res64;      // ||b||, the recurrence's ||r||, ||b - A x||
    int it, breakdown;
    int unfit;                 // a block's rows do not fit its shared memory: nothing was solved
    int timeout;               // a block waited past the bound for the others
};

struct ResidentPlan {
    bool cluster = false;      // one thread-block cluster (its barrier, distributed shared memory)
    int blocks = 0, smem = 0;
};

static constexpr int RES_MAX_BLOCKS = 256;
// the solve's scratch: n doubles of exchanged vector, the blocks' sums and their counter, the result
static constexpr size_t RES_SUM_DOUBLES = 2 * 3 * RES_MAX_BLOCKS, RES_SLOT_DOUBLES = RES_SUM_DOUBLES + 2;
static constexpr size_t RES_OUT_DOUBLES = (sizeof(ResidentOut) + sizeof(double) - 1) / sizeof(double);

// Whether (and how) a system of n rows and nnz entries is solved on chip; unfit: the forms that were found
// not to hold it.
static constexpr int RES_UNFIT_CLUSTER = 1, RES_UNFIT_GRID = 2;
bool resident_plan(femd_ctx ctx, int n, long long nnz, int unfit, ResidentPlan &plan);

// One solve on the stream: x is read as the start and holds the solution; inv may be null (no
// preconditioner). zx: n doubles; slots: RES_SLOT_DOUBLES doubles; out: device.
cudaError_t resident_launch(const ResidentPlan &plan, const int *indptr, const int *indices, const double *data,
                            const double *inv, const double *b, double *x, int n, int max_iter, double tol, double *zx,
                            double *slots, ResidentOut *out, cudaStream_t s);

}  // namespace femd
