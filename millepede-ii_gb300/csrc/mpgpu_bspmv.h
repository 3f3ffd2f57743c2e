// mpgpu_bspmv.h -- symmetric product of the mpbits-sparse global matrix from
// a block-row copy (mpgpu_bspmv.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "mpgpu_minres.cuh"

struct mpgpu_ctx;
struct DevJob;

// Device arrays of the copy, kept (with their capacities) in the job between
// the solves of a layout.
struct BlockRows {
    int R = 0;                    // padded parameters per group (1..8); 0: not built
    int nslot = 0;                // blocks per step: 32 / R
    int32_t nG = 0, nVar = 0;
    int64_t nsteps = 0, nitem = 0;
    bool uniform = true;          // every group has R parameters: padded index = index
    double *val = nullptr;        // [nsteps][R][nslot * R], element pairs for even R
    int32_t *col = nullptr;       // [nsteps * nslot] column group, 0-based
    int64_t *stepBeg = nullptr;   // [nG + 1]
    int64_t *itemBeg = nullptr;   // [nG + 1]
    int32_t *itemS0 = nullptr, *itemS1 = nullptr;   // [nitem] steps of the item
    double *part = nullptr;       // [nitem * R]
    double *xp = nullptr;         // [nG * R] padded vector
};

// Whether the copy serves this layout: sparse storage, groups of at most 8
// parameters, little padding.
bool block_rows_fit(const mpgpu_ctx *c);
// Builds the copy of the current matrix on the context's stream (in the job's br).
int32_t block_rows_build(mpgpu_ctx *c);
// its device memory, and giving it back
int64_t block_rows_bytes(const BlockRows &b);
void block_rows_free(DevJob &j);
// part = item sums of A xp (xp padded: parameter i of group g at g R + i); nothing
// when *done is set.  coef: work of one extra CTA (null: none)
struct BlockRowsCoef {
    int32_t m;                // constraints
    int32_t nblk;             // partial dots per column
    const double *partUW;     // [nblk][2 m] partial sums of x with the columns [U | W]
    const double *T, *S;      // m x m: compact WY factor, T (U^T A U) T^T
    double *coef;             // [2 m] c (of U), a (of W)
    MinresTest test;          // of the last iteration, taken by the same CTA
};
cudaError_t block_rows_spmv(const BlockRows &b, const double *xp, const int32_t *done, const BlockRowsCoef *coef,
                            cudaStream_t s);
// y = A x of whole vectors of nVar elements (pads x, sums the items)
cudaError_t block_rows_product(const BlockRows &b, const int32_t *aig, const int32_t *p2g, const double *x, double *y,
                               cudaStream_t s);
