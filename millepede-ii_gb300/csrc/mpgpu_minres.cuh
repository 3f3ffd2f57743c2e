// mpgpu_minres.cuh -- iteration scalars of the device MINRES / MINRES-QLP
// (mpgpu_solve.cu) and their convergence test, which rides in the extra CTA
// of the block-row product (mpgpu_bspmv.cu).
#pragma once
#include <cuda_runtime.h>

// Two copies alternate from iteration to iteration: the kernel that takes
// the scalar step (k_mr_step) computes it in every CTA from one copy and
// writes the other, so no CTA reads what another one is writing.
struct MinresState {
    double beta1, beta, oldb, alfa, dbar, epsln, oldeps, delta, gbar, cs, sn, phi, phibar;
    double tnorm2, gmax, gmin, Anorm, ynorm, rnorm, denom, rtol;
    double invb, bo;              // 1 / beta, beta / oldb
    int k;                        // iterations whose update is done
    int itn, itnlim, istop;
};

// done: the last test ended the iteration; commit: it accepted the
// candidate iterate of MINRES-QLP.  alfa stands between k_mr_y2 and the
// scalar step.
struct MinresFlags {
    int done, commit;
    double alfa;
};

// Convergence test of the last update from x . x (partial sums partX): one
// CTA, of which the first warp works.  maxxnorm < 0: MINRES.
struct MinresTest {
    MinresState *S;
    MinresFlags *F;
    const double *partX;
    int npX;
    double maxxnorm;
};

// sum of n values in a fixed order by one warp, in every lane
__device__ __forceinline__ double warp_sum_of(const double *part, int n) {
    double v = 0.0;
#pragma unroll 8
    for (int i = threadIdx.x & 31; i < n; i += 32) v += part[i];
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    return v;
}

__device__ inline void mr_test(const MinresTest &t) {
    if (threadIdx.x >= 32) return;
    MinresState *S = t.S;
    const int k = S->k;
    if (k <= 0) return;
    if (S->istop == 9) {
        if (threadIdx.x == 0) {
            t.F->commit = 0;
            t.F->done = 1;
        }
        return;
    }
    const double xx = warp_sum_of(t.partX, t.npX);
    if (threadIdx.x) return;
    const double xnorm = sqrt(xx), Anorm = sqrt(S->tnorm2), rnorm = S->phibar;
    const bool commit = !(t.maxxnorm >= 0.0 && xnorm > t.maxxnorm);
    const double root = sqrt(S->gbar * S->gbar + S->dbar * S->dbar);
    const double test1 = rnorm / (Anorm * xnorm), test2 = root / Anorm;
    int istop = 0;
    if (k >= S->itnlim) istop = 6;
    if (S->gmax / S->gmin >= 0.1 / 2.220446049250313e-16) istop = 4;
    if (test2 <= S->rtol) istop = 2;
    if (test1 <= S->rtol) istop = 1;
    if (!commit) istop = 5;
    S->itn = k;
    if (commit) {
        S->Anorm = Anorm;
        S->ynorm = xnorm;
        S->rnorm = rnorm;
    }
    t.F->commit = commit;
    if (istop) {
        S->istop = istop;
        t.F->done = 1;
    }
}
