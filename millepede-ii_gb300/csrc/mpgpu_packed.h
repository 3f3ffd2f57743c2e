// mpgpu_packed.h -- factorisations of the packed symmetric matrix on the
// device (mpgpu_packed.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

// doubles of workspace for an n x n leading block
int64_t packed_work_len(int32_t n);
// sqminl (mpnum.f90:230-355): V (packed, leading n x n block) is replaced by
// minus the swept matrix, b by the solution; diag[n]: |original diagonal|;
// used[n] receives the pivoted rows.  *deficit is -1 when no pivot was left
// before all rows were used, else 0.
cudaError_t packed_sqminl(int32_t n, double *V, double *b, const double *diag, int32_t *used, int32_t *deficit,
                          double *work, cudaStream_t s);
// chdec2 + chslv2 (mpnum.f90:891-987): g (packed) is decomposed, x solved.
// stat: largest pivot, smallest pivot, number of positive pivots (zeroed by
// the caller).
cudaError_t packed_chdec_solve(int32_t n, double *g, double *x, double *stat, double *work, cudaStream_t s);
