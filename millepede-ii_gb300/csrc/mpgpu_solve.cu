// mpgpu_solve.cu -- global solvers on the device: QL constraint
// elimination products, packed Gauss-Jordan inversion (sqminl), root-free
// Cholesky (chdec2/chslv2), the sparse and packed symmetric matrix-vector
// product (avprd0) and preconditioned MINRES.  All reductions have a fixed
// shape, so repeated solves give bit-identical results.
#include <cuda_runtime.h>

#include <algorithm>
#include <cmath>
#include <cstring>
#include <vector>

#include "mpgpu_bspmv.h"
#include "mpgpu_ctx.h"
#include "mpgpu_packed.h"

namespace {

constexpr int kDotBlocks = 304;   // 2 x 152 SMs, fixed for determinism
constexpr int kThreads = 256;

template <class T>
void dfree(T *&p) {
    if (p) cudaFree(p);
    p = nullptr;
}

// ---------------------------------------------------------------- reductions
__device__ __forceinline__ double block_sum(double v, double *sh) {
    sh[threadIdx.x] = v;
    __syncthreads();
    for (int s = blockDim.x / 2; s > 0; s >>= 1) {
        if ((int)threadIdx.x < s) sh[threadIdx.x] += sh[threadIdx.x + s];
        __syncthreads();
    }
    double r = sh[0];
    __syncthreads();
    return r;
}

__global__ void k_dot_partial(int64_t n, const double *a, const double *b, double *part) {
    __shared__ double sh[kThreads];
    double s = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        s += a[i] * b[i];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) part[blockIdx.x] = s;
}

__global__ void k_sum_final(const double *part, int n, double *out) {
    __shared__ double sh[kThreads];
    double s = 0.0;
    for (int i = threadIdx.x; i < n; i += blockDim.x) s += part[i];
    s = block_sum(s, sh);
    if (threadIdx.x == 0) *out = s;
}

void dot(const double *a, const double *b, int64_t n, double *part, double *out, cudaStream_t s) {
    k_dot_partial<<<kDotBlocks, kThreads, 0, s>>>(n, a, b, part);
    k_sum_final<<<1, kThreads, 0, s>>>(part, kDotBlocks, out);
}

// ---------------------------------------------------------------- QL products
// qlmlq (mpqldec.f90:404-454) for one vector, one CTA walking the
// reflections k = kfirst, kfirst+step, ..., klast in that order
// (Q x: 1..ncon; Q^T x: ncon..1).
__global__ void k_qlapply(double *x, const double *V, const double *Vk, const int32_t *r2, int32_t npar,
                          int32_t ncon, int kfirst, int klast, int step) {
    __shared__ double sh[1024];
    if (step == 0) return;
    for (int k = kfirst; step > 0 ? k <= klast : k >= klast; k += step) {
        const int kn = npar + k - ncon;
        const int ilast = r2[k - 1];
        const double *v = V + (int64_t)(k - 1) * npar;
        const double vk = Vk[k - 1];
        double s = 0.0;
        for (int i = threadIdx.x; i < ilast; i += blockDim.x) s += v[i] * x[i];
        s = block_sum(s, sh);
        const double sp = s + vk * x[kn - 1];
        __syncthreads();
        for (int i = threadIdx.x; i < ilast; i += blockDim.x) x[i] = x[i] - 2.0 * v[i] * sp;
        if (threadIdx.x == 0) x[kn - 1] = x[kn - 1] - 2.0 * vk * sp;
        __syncthreads();
    }
}

// qlmlq in the compact WY form: Q^T x = x - U T (U^T x), Q x = x - U T^T
// (U^T x), U = the reflection vectors (rows of V with Vk at position
// npar - ncon + k).  Pass 1: per CTA the partial products of eight vectors
// at a time over a fixed row partition; pass 2 (one CTA): the sums in CTA
// order plus the Vk terms, then t = T s or T^T s; pass 3: x -= U t.
constexpr int kWyBlocks = 304;

__global__ void __launch_bounds__(256) k_wy_dots(int32_t n, int32_t m, const double *V, const double *x,
                                                  double *part) {
    __shared__ double sh[8][8];
    const int ln = threadIdx.x & 31, wib = threadIdx.x >> 5;
    for (int32_t k0 = 0; k0 < m; k0 += 8) {
        const int kc = min(8, m - k0);
        double acc[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) acc[q] = 0.0;
        for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
            const double xi = x[i];
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (q < kc) acc[q] += V[(int64_t)(k0 + q) * n + i] * xi;
        }
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            double v = acc[q];
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (ln == 0) sh[q][wib] = v;
        }
        __syncthreads();
        if ((int)threadIdx.x < kc) {
            double v = 0.0;
            for (int w8 = 0; w8 < (int)(blockDim.x >> 5); ++w8) v += sh[threadIdx.x][w8];
            part[(int64_t)blockIdx.x * m + k0 + threadIdx.x] = v;
        }
        __syncthreads();
    }
}

__global__ void k_wy_coef(int32_t n, int32_t m, int32_t nblk, const double *part, const double *Vk,
                          const double *T, const double *x, int transT, double *tv) {
    extern __shared__ double sv[];
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
        double s = 0.0;
        for (int b = 0; b < nblk; ++b) s += part[(int64_t)b * m + k];
        sv[k] = s + Vk[k] * x[n - m + k];
    }
    __syncthreads();
    for (int k = threadIdx.x; k < m; k += blockDim.x) {
        double t = 0.0;
        if (transT)
            for (int c = 0; c <= k; ++c) t += T[(int64_t)c * m + k] * sv[c];
        else
            for (int c = k; c < m; ++c) t += T[(int64_t)k * m + c] * sv[c];
        tv[k] = t;
    }
}

__global__ void k_wy_apply(int32_t n, int32_t m, const double *V, const double *Vk, const double *tv, double *x) {
    extern __shared__ double st[];
    for (int k = threadIdx.x; k < m; k += blockDim.x) st[k] = tv[k];
    __syncthreads();
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        double a = 0.0;
        for (int k = 0; k < m; ++k) a += V[(int64_t)k * n + i] * st[k];
        const int64_t kk = i - (n - m);
        if (kk >= 0) a += Vk[kk] * st[kk];
        x[i] -= a;
    }
}

// ---------------------------------------------------------------- packed products
// y = A x for the packed symmetric matrix in two deterministic passes.
// Pass 1, one CTA per 16 rows x 1,024 columns, a thread per column: every
// element is read once and used for its row's sum and for its column's.  Pass 2
// adds, per j, the row parts by column range and the column parts of the blocks
// below j, eight threads per j.
// FP64-bound: two multiply-adds per stored element (57 us for 6,000 rows; the
// matrix once takes 22 us).  Reading it once per row and once per column took
// 248 + 85 us, now 99 + 15 (1,500 rows: 21 + 14 us, now 20 + 4).
constexpr int kMvRows = 16;
constexpr int kMvCols = 1024;

// sums of v[0..15] over the warp, v[r] in lanes 2 r and 2 r + 1
__device__ __forceinline__ double warp_sum16(double (&v)[kMvRows]) {
    const int ln = threadIdx.x & 31;
#pragma unroll
    for (int h = kMvRows / 2; h > 0; h >>= 1) {
        const bool up = ln & (2 * h);
#pragma unroll
        for (int r = 0; r < h; ++r) {
            const double give = up ? v[r] : v[r + h];
            const double keep = up ? v[r + h] : v[r];
            v[r] = keep + __shfl_xor_sync(0xffffffffu, give, 2 * h);
        }
    }
    return v[0] + __shfl_xor_sync(0xffffffffu, v[0], 1);
}

__global__ void __launch_bounds__(256, 3) k_pmv_blocks(int32_t n, const double *A, const double *x, double *yrow,
                                                     double *part) {
    __shared__ double xs[kMvRows], ws[8][kMvRows];
    const int64_t b = gridDim.x - 1 - blockIdx.x;   // the longest rows first
    const int64_t i0 = b * kMvRows, i1 = min((int64_t)n, i0 + kMvRows), j0 = (int64_t)blockIdx.y * kMvCols;
    if (j0 >= i1) return;
    const int tid = threadIdx.x, ln = tid & 31, wib = tid >> 5;
    if (tid < kMvRows) xs[tid] = i0 + tid < n ? x[i0 + tid] : 0.0;
    __syncthreads();
    const int64_t j1 = min(i1, j0 + kMvCols);
    const double *base = A + i0 * (i0 + 1) / 2;
    double r[kMvRows] = {};
    for (int64_t j = j0 + tid; j < j1; j += 256) {
        const double xj = x[j];
        double a[kMvRows], c = 0.0;
        if (j < i0 && i1 == i0 + kMvRows) {
#pragma unroll
            for (int q = 0; q < kMvRows; ++q) a[q] = base[q * i0 + q * (q + 1) / 2 + j];
#pragma unroll
            for (int q = 0; q < kMvRows; ++q) {
                r[q] = fma(a[q], xj, r[q]);
                c = fma(a[q], xs[q], c);
            }
        } else {
#pragma unroll
            for (int q = 0; q < kMvRows; ++q) {
                a[q] = (i0 + q < i1 && j <= i0 + q) ? base[q * i0 + q * (q + 1) / 2 + j] : 0.0;
                if (i0 + q < i1 && j <= i0 + q) r[q] = fma(a[q], xj, r[q]);
                if (i0 + q < i1 && j < i0 + q) c = fma(a[q], xs[q], c);
            }
        }
        if (j < i1 - 1) part[b * (int64_t)n + j] = c;
    }
    const double t = warp_sum16(r);
    // lane bits 4..1 select the row: bit 4 the upper half, ...
    if (!(ln & 1)) ws[wib][ln >> 1] = t;
    __syncthreads();
    if (tid < kMvRows && i0 + tid < i1) {
        double sum = ws[0][tid];
#pragma unroll
        for (int w = 1; w < 8; ++w) sum += ws[w][tid];
        yrow[blockIdx.y * (int64_t)n + i0 + tid] = sum;
    }
}

__global__ void __launch_bounds__(256) k_pmv_final(int32_t n, int64_t nb, const double *yrow, const double *part,
                                                   double *y) {
    __shared__ double ps[8][32];
    const int ln = threadIdx.x & 31, wib = threadIdx.x >> 5;
    const int64_t j = (int64_t)blockIdx.x * 32 + ln;
    double s = 0.0;
    if (j < n) {
        for (int64_t b = (j + 1) / kMvRows + wib; b < nb; b += 8) {
            const int64_t i1 = min((int64_t)n, (b + 1) * kMvRows);
            if (j < i1 - 1) s += part[b * (int64_t)n + j];
        }
    }
    ps[wib][ln] = s;
    __syncthreads();
    if (wib == 0 && j < n) {
        double t = yrow[j];
        // row j's CTA covers all columns of its block of rows
        const int64_t last = min((int64_t)n, (j / kMvRows + 1) * kMvRows) - 1;
        for (int64_t q = 1; q <= last / kMvCols; ++q) t += yrow[q * (int64_t)n + j];
#pragma unroll
        for (int w = 0; w < 8; ++w) t += ps[w][ln];
        y[j] = t;
    }
}

// qlssq update of one reflection on the packed matrix (mpqldec.f90:
// 644-686): rows 1..kn get 2(2 v_i vtAv - Av_i) v_c for c in [1, min(ilast,i)],
// rows ilast and below in [1, ilast] get -2 Av_c v_i, the diagonal (kn,kn)
// its combined term and rows > kn their -2 v_c Av_i parts.  Tiles of 16 rows x
// 256 columns, a thread per column: the row's and the column's factors are
// read once per tile.  FP64-bound: two multiply-adds per element (57 us for
// 6,000 rows, reading and writing the matrix 43 us); a warp per row took 210
// us, now 104.
constexpr int kQlRows = 16;
constexpr int kQlCols = 256;
__global__ void __launch_bounds__(256, 2) k_qlssq_update(int32_t n, double *A, const double *v, double vk,
                                                      const double *Av, const double *vtAvp, int32_t ilast,
                                                      int32_t kn) {
    __shared__ double fa[kQlRows], fb[kQlRows];
    const int64_t i0 = (int64_t)(gridDim.x - 1 - blockIdx.x) * kQlRows, j0 = (int64_t)blockIdx.y * kQlCols;   // 0-based
    const int64_t i1 = min((int64_t)n, i0 + kQlRows);
    if (j0 >= i1) return;
    const double vtAv = *vtAvp;
    const int tid = threadIdx.x;
    if (tid < kQlRows && i0 + tid < i1) {
        const int64_t i = i0 + tid + 1;   // 1-based
        const double vi = i <= ilast ? v[i - 1] : (i == kn ? vk : 0.0), av = Av[i - 1];
        fa[tid] = i <= kn ? 2.0 * (2.0 * vi * vtAv - av) : -2.0 * av;   // times v_c
        fb[tid] = -2.0 * vi;                                           // times Av_c, rows up to ilast
    }
    __syncthreads();
    double *base = A + i0 * (i0 + 1) / 2;
    const int64_t j1 = min(min(i1, j0 + kQlCols), (int64_t)ilast);
    for (int64_t j = j0 + tid; j < j1; j += 256) {
        const double vc = v[j], ac = Av[j];
        if (j < i0 && i1 == i0 + kQlRows && i1 <= ilast) {
            double a[kQlRows];
#pragma unroll
            for (int q = 0; q < kQlRows; ++q) a[q] = base[q * i0 + q * (q + 1) / 2 + j];
#pragma unroll
            for (int q = 0; q < kQlRows; ++q)
                base[q * i0 + q * (q + 1) / 2 + j] = fma(fb[q], ac, fma(fa[q], vc, a[q]));
        } else {
            for (int q = 0; q < (int)(i1 - i0); ++q) {
                if (j > i0 + q) continue;
                double *p = base + q * i0 + q * (q + 1) / 2 + j;
                double a = fma(fa[q], vc, *p);
                if (i0 + q < ilast) a = fma(fb[q], ac, a);
                *p = a;
            }
        }
    }
    // column kn: the diagonal element and the rows below it
    if (tid < (int)(i1 - i0) && kn - 1 >= j0 && kn - 1 < j0 + kQlCols) {
        const int64_t i = i0 + tid + 1;
        double *p = base + tid * i0 + tid * (tid + 1) / 2 + kn - 1;
        if (i == kn) *p = *p + 2.0 * ((2.0 * vk * vtAv - Av[kn - 1]) * vk - Av[kn - 1] * vk);
        if (i > kn) *p = *p - 2.0 * vk * Av[i - 1];
    }
}

__global__ void k_vec_with_kn(const double *v, int32_t ilast, double vk, int32_t kn, int32_t n, double *out) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        out[i] = i < ilast ? v[i] : (i == kn - 1 ? vk : 0.0);
}

// sqminl without a pivot left: rows and columns of the unused rows zeroed
__global__ void k_sqminl_deficit(int32_t n, double *v, double *b, const int32_t *used, const int32_t *pivot) {
    if (*pivot >= 0) return;
    for (int64_t j = blockIdx.x; j < n; j += gridDim.x) {
        if (used[j]) continue;
        if (threadIdx.x == 0) b[j] = 0.0;
        double *row = v + j * (j + 1) / 2;
        for (int64_t c = threadIdx.x; c <= j; c += blockDim.x)
            if (!used[c]) row[c] = 0.0;
    }
}

__global__ void k_negate(int64_t n, double *v) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        v[i] = -v[i];
}

__global__ void k_diag_abs(int32_t n, const double *v, double *d) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        d[i] = fabs(v[(i + 1) * (i + 2) / 2 - 1]);
}

// corr(i) -= sum_j A'(nfit+j, i) y(j), i <= nfit (minver/mchdec rhs)
__global__ void k_cons_rhs(int32_t nfit, int32_t ncon, const double *A, const double *y, double *corr) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < nfit; i += (int64_t)gridDim.x * blockDim.x) {
        double cval = corr[i];
        for (int j = 0; j < ncon; ++j) {
            const int64_t r = nfit + j + 1;
            cval = cval - A[(r * r - r) / 2 + i] * y[j];
        }
        corr[i] = cval;
    }
}

__global__ void k_zero_rows(int32_t nfit, int32_t n, double *A) {
    for (int64_t r = nfit + 1 + blockIdx.x; r <= n; r += gridDim.x) {
        double *row = A + (r * r - r) / 2;
        for (int64_t c = threadIdx.x; c < r; c += blockDim.x) row[c] = 0.0;
    }
}

__global__ void k_get_diag(int32_t n, const double *A, double *d) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        d[i] = A[(i + 1) * (i + 2) / 2 - 1];
}

// ---------------------------------------------------------------- sparse SpMV
// Block table of the mpbits storage: for every stored block (I, J <= I) the
// 0-based offset of element (0,0) in globalMatD and the row stride.
struct SparseBlocks {
    int64_t nblk = 0;
    int64_t *rowStart = nullptr;   // [nG+1] blocks of row group I
    int32_t *bcol = nullptr;       // column group
    int64_t *boff = nullptr;
    int32_t *bld = nullptr;
    int64_t *tOff = nullptr;       // transposed-product buffer offset (off-diagonal blocks)
    int64_t *colStart = nullptr;   // [nG+1] incoming blocks of column group J
    int64_t *colBlk = nullptr;     // block ids ordered by (J, I)
    int64_t *tBase = nullptr;      // [nG] first transposed product of column group J
    double *tbuf = nullptr;
    int64_t tlen = 0;
    bool smallGroups = false;     // every group has at most kSmallGroup parameters
    // small groups: per block its row group (brow), its partial row sums
    // (rowPart, kSmallGroup each) and the stride of its transposed products
    // (tStr: the column group's incoming block count, parameter-major)
    int32_t *brow = nullptr;       // [nblk]
    int32_t *tStr = nullptr;       // [nblk]
    double *rowPart = nullptr;     // [nblk * kSmallGroup]
    // column items: at most kColItem incoming blocks of one column group
    int64_t nColItem = 0;
    int32_t *colItemJ = nullptr;   // [nColItem]
    int64_t *colItemQ0 = nullptr;  // [nColItem] first incoming block (0-based within the group)
    int64_t *colItemQ1 = nullptr;  // [nColItem] end
    int64_t *colItemBeg = nullptr; // [nG+1] first item of column group J
    double *colPart = nullptr;     // [nColItem * kSmallGroup]
    int uniform = 0;               // every group has this many parameters (0: mixed)
};

// phase 1: warp per row group I: y_I = D_I x_I + sum_J A_IJ x_J, the
// strictly-lower part of the diagonal block also transposed into y_I, and
// t_IJ = A_IJ^T x_I for J < I into tbuf
__global__ void k_spmv_rows(int32_t nG, const int32_t *aig, const int64_t *rowStart, const int32_t *bcol,
                            const int64_t *boff, const int32_t *bld, const int64_t *tOff,
                            const double *matD, const double *x, double *y, double *tbuf) {
    const int ln = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t I = 1 + w; I <= nG; I += nw) {
        const int32_t ia = aig[I - 1] - 1, np = aig[I] - 1 - ia;
        for (int ii = 0; ii < np; ++ii) {
            double s = 0.0;
            for (int64_t bl = rowStart[I - 1]; bl < rowStart[I]; ++bl) {
                const int32_t J = bcol[bl];
                const int32_t ja = aig[J - 1] - 1, nj = aig[J] - 1 - ja;
                const double *row = matD + boff[bl] + (int64_t)ii * bld[bl];
                if (J == I) {
                    for (int jj = ln; jj < ii; jj += 32) s += row[jj] * x[ja + jj];
                    // transposed strictly-lower part: A(r, ii) for r > ii
                    for (int rr = ii + 1 + ln; rr < np; rr += 32)
                        s += matD[boff[bl] + (int64_t)rr * bld[bl] + ii] * x[ia + rr];
                } else {
                    for (int jj = ln; jj < nj; jj += 32) s += row[jj] * x[ja + jj];
                }
            }
            for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
            if (ln == 0) y[ia + ii] = matD[ia + ii] * x[ia + ii] + s;
        }
        // transposed products of the off-diagonal blocks
        for (int64_t bl = rowStart[I - 1]; bl < rowStart[I]; ++bl) {
            const int32_t J = bcol[bl];
            if (J == I) continue;
            const int32_t nj = aig[J] - aig[J - 1];
            for (int jj = ln; jj < nj; jj += 32) {
                double t = 0.0;
                for (int ii = 0; ii < np; ++ii) t += matD[boff[bl] + (int64_t)ii * bld[bl] + jj] * x[ia + ii];
                tbuf[tOff[bl] + jj] = t;
            }
        }
    }
}

// phase 2: warp per column group J adds the transposed products in a fixed order
__global__ void k_spmv_cols(int32_t nG, const int32_t *aig, const int64_t *colStart, const int64_t *colBlk,
                            const int64_t *tOff, const double *tbuf, double *y) {
    const int ln = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t J = 1 + w; J <= nG; J += nw) {
        const int32_t ja = aig[J - 1] - 1, nj = aig[J] - 1 - ja;
        for (int jj = ln; jj < nj; jj += 32) {
            double s = y[ja + jj];
            for (int64_t q = colStart[J - 1]; q < colStart[J]; ++q) s += tbuf[tOff[colBlk[q]] + jj];
            y[ja + jj] = s;
        }
    }
}

// the same two phases for row groups of at most 8 parameters of strongly
// mixed sizes, or where the memory does not hold the block-row copy that the
// others take (mpgpu_bspmv.cu).  Phase 1,
// one thread per stored block (all blocks of all row groups, so the lanes
// stay full whatever the row lengths): the block's rows times x_J into its
// partial row sums (rowPart, 8 per block; the diagonal block adds both
// triangles of its strictly-lower part there) and its columns times x_I
// into tbuf (parameter-major per column group).  G > 0: every group has G
// parameters (loops fully unrolled); G = 0: at most 8, predicated.  Phase 2:
// the partial row sums of a group's blocks and the transposed products of its
// incoming blocks summed by column items (long columns split over several
// warps), then y = D x + the group's items in item order; no atomics, the sums
// are reproducible.
constexpr int kSmallGroup = 8;

template <int G>
__global__ void __launch_bounds__(256) k_spmv_blocks(int64_t nb, const int32_t *brow, const int32_t *aig,
                                                     const int32_t *bcol, const int64_t *boff, const int32_t *bld,
                                                     const int64_t *tOff, const int32_t *tStr,
                                                     const double *matD, const double *x, double *tbuf,
                                                     double *rowPart) {
    constexpr int M = G > 0 ? G : kSmallGroup;
    for (int64_t bl = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; bl < nb;
         bl += (int64_t)gridDim.x * blockDim.x) {
        const int32_t I = brow[bl], J = bcol[bl];
        const int32_t ia = aig[I - 1] - 1, ja = aig[J - 1] - 1;
        const int np = G > 0 ? G : aig[I] - 1 - ia;
        const int nj = G > 0 ? G : aig[J] - 1 - ja;
        const double *blk = matD + boff[bl];
        const int32_t ld = bld[bl];
        double xi[M], sr[M];
#pragma unroll
        for (int ii = 0; ii < M; ++ii) {
            xi[ii] = ii < np ? x[ia + ii] : 0.0;
            sr[ii] = 0.0;
        }
        if (J != I) {
            double xj[M], tc[M];
#pragma unroll
            for (int jj = 0; jj < M; ++jj) {
                xj[jj] = jj < nj ? x[ja + jj] : 0.0;
                tc[jj] = 0.0;
            }
#pragma unroll
            for (int ii = 0; ii < M; ++ii) {
                if (ii < np) {
#pragma unroll
                    for (int jj = 0; jj < M; ++jj) {
                        if (jj < nj) {
                            const double a = blk[(int64_t)ii * ld + jj];
                            sr[ii] += a * xj[jj];
                            tc[jj] += a * xi[ii];
                        }
                    }
                }
            }
            double *tb = tbuf + tOff[bl];
            const int32_t st = tStr[bl];
#pragma unroll
            for (int jj = 0; jj < M; ++jj)
                if (jj < nj) tb[(int64_t)jj * st] = tc[jj];
        } else {
#pragma unroll
            for (int ii = 1; ii < M; ++ii) {
                if (ii < np) {
#pragma unroll
                    for (int jj = 0; jj < ii; ++jj) {
                        const double a = blk[(int64_t)ii * ld + jj];
                        sr[ii] += a * xi[jj];
                        sr[jj] += a * xi[ii];
                    }
                }
            }
        }
        double *rp = rowPart + bl * kSmallGroup;
#pragma unroll
        for (int ii = 0; ii < M; ++ii) rp[ii] = sr[ii];
    }
}

// phase 2a, one warp per column item (at most kColItem incoming blocks of
// one column group; the first item of a group also takes the partial row
// sums of the group's own blocks): lanes with four independent partial
// sums, a fixed shuffle tree, into colPart (8 per item)
constexpr int kColItem = 128;

__global__ void __launch_bounds__(256) k_spmv_colitems(int64_t nItem, const int32_t *itemJ, const int64_t *itemQ0,
                                                       const int64_t *itemQ1, const int32_t *aig,
                                                       const int64_t *rowStart, const double *rowPart,
                                                       const int64_t *colStart, const int64_t *tBase,
                                                       const double *tbuf, double *colPart) {
    const int ln = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t it = w; it < nItem; it += nw) {
        const int32_t J = itemJ[it];
        const int32_t nj = aig[J] - aig[J - 1];
        const int64_t q0 = itemQ0[it], q1 = itemQ1[it];
        const bool first = q0 == 0;
        const int64_t r0 = rowStart[J - 1], nr = first ? rowStart[J] - r0 : 0;
        const int64_t cnt = colStart[J] - colStart[J - 1];
        const double *t = tbuf + tBase[J - 1];
        for (int jj = 0; jj < kSmallGroup; ++jj) {
            double v = 0.0;
            if (jj < nj) {
                double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
                for (int64_t q = ln; q < nr; q += 32) v0 += rowPart[(r0 + q) * kSmallGroup + jj];
                const double *tj = t + (int64_t)jj * cnt;
                int64_t q = q0 + ln;
                for (; q + 96 < q1; q += 128) {
                    v0 += tj[q];
                    v1 += tj[q + 32];
                    v2 += tj[q + 64];
                    v3 += tj[q + 96];
                }
                for (; q < q1; q += 32) v1 += tj[q];
                v = (v0 + v1) + (v2 + v3);
            }
            for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
            if (ln == 0) colPart[it * kSmallGroup + jj] = v;
        }
    }
}

// phase 2b, one thread per parameter: y = D x + the column items of its
// group in item order
__global__ void k_spmv_final(int32_t n, const int32_t *aig, const int32_t *p2g, const int64_t *colItemBeg,
                             const double *colPart, const double *matD, const double *x, double *y) {
    for (int64_t j = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; j < n; j += (int64_t)gridDim.x * blockDim.x) {
        const int32_t J = p2g[j];
        const int32_t jj = (int32_t)j - (aig[J - 1] - 1);
        double r = matD[j] * x[j];
        for (int64_t it = colItemBeg[J - 1]; it < colItemBeg[J]; ++it) r += colPart[it * kSmallGroup + jj];
        y[j] = r;
    }
}

// ---------------------------------------------------------------- MINRES state
// MINRES-QLP (Choi, Paige & Saunders 2011; minresqlpModule.f90:411-1333 in
// the reference): the Lanczos scalars of MinresState plus the rows of the
// lower-triangular L = R P not yet final, the final u values and the
// rotations of the current iteration for the vector kernel
struct QlpState {
    double etaA, thA, gA, tauA, etaB, thB, gB, tauB, uF1, uF2;
    double c1, s1, c2, s2, uA, uB, uC;
};

// sum over the CTA (T threads) in a fixed order, in thread 0; sh: T / 32
template <int T>
__device__ __forceinline__ double cta_sum(double v, double *sh) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
    if ((threadIdx.x & 31) == 0) sh[threadIdx.x >> 5] = v;
    __syncthreads();
    double r = sh[0];
    if (threadIdx.x == 0) {
#pragma unroll
        for (int q = 1; q < T / 32; ++q) r += sh[q];
    }
    return r;
}

// beta1^2 = r1 . y
__global__ void k_mr_init(MinresState *S, QlpState *Q, MinresFlags *F, const double *dotv, double rtol, int itnlim) {
    if (threadIdx.x) return;
    memset(S, 0, 2 * sizeof(MinresState));
    if (Q) memset(Q, 0, 2 * sizeof(QlpState));
    F->done = F->commit = 0;
    S->rtol = rtol;
    S->itnlim = itnlim;
    S->cs = -1.0;
    S->gmin = 1.0e300;
    double b1 = *dotv;
    if (b1 <= 0.0) { S->istop = b1 < 0.0 ? 9 : 0; F->done = 1; return; }
    b1 = sqrt(b1);
    S->beta1 = b1;
    S->beta = b1;
    S->invb = 1.0 / b1;
    S->phibar = b1;
}

// One iteration is four launches: operator product with the convergence
// test of the last update beside it (block_rows_spmv; k_mr_test and the
// separate products of the other storages), k_mr_y1, k_mr_y2, k_mr_step.
// The dot products that end one kernel are summed by every CTA of the next
// one (at most kMrBlocks values).  They are bound by launch and
// synchronisation latency, not by their 0.2 MB vectors, and by FP64
// instructions that every warp would repeat (a warp's FP64 instruction holds
// its quarter of the SM for 64 clocks, and a division is about 30 of them), so
// the scalars are formed by one warp.  At 30,000 globals and 18 constraints: product 35 to
// 44 us (mpgpu_bspmv.cu), 9.8, 6.2 and 10.9 us.  The first form had 16
// launches, with the sums in kernels of one CTA.
constexpr int kMrBlocks = 1216;    // CTAs of the vector kernels (at most)
constexpr int kY1Threads = 512, kY1Lanes = 4;   // k_mr_y1: lanes per row
constexpr int kStepRows = 128;     // rows per round of k_mr_step
constexpr int kStepBlocks = 304;
constexpr int kWyFused = 64;       // constraints whose products ride in the iteration's kernels

// the test alone (paths without block_rows_spmv's extra CTA)
__global__ void k_mr_test(MinresTest t) {
    if (t.F->done) return;
    mr_test(t);
}

// y = Q^T A Q v on the fitted rows: with the block-row copy the item sums
// less [U | W] coef (coef of br_coef), else the separate products' ba; then
// y -= (beta / oldbeta) r1 from the second iteration on, partials of v . y.
// With xc, the MINRES-QLP iterate that the test has just accepted is
// committed first.  kY1Lanes lanes share a row's items and columns: one lane
// per row waits for about ten dependent loads in a row of 20 items and 36
// columns (14.2 us, 9.8 us with four).
struct Y1Params {
    int32_t nfit, n, m, R;
    const int32_t *aig, *p2g;
    const int64_t *itemBeg;
    const double *part, *UWc, *coef, *ba, *r1, *v, *xc;
    const MinresState *S;
    const MinresFlags *F;
    double *y, *x, *partA;
};

template <bool ITEMS>
__global__ void __launch_bounds__(kY1Threads) k_mr_y1(Y1Params p) {
    constexpr int L = kY1Lanes;
    __shared__ double sh[kY1Threads / 32], cs[2 * kWyFused];
    const int64_t t0 = (int64_t)blockIdx.x * kY1Threads + threadIdx.x, step = (int64_t)gridDim.x * kY1Threads;
    if (p.xc && p.F->commit)
        for (int64_t i = t0; i < p.nfit; i += step) p.x[i] = p.xc[i];
    if (p.F->done) return;
    const int C = ITEMS ? 2 * p.m : 0;
    if ((int)threadIdx.x < C) cs[threadIdx.x] = p.coef[threadIdx.x];
    __syncthreads();
    const bool upd = p.S->k >= 1;
    const double f = p.S->bo;
    const int sub = threadIdx.x % L;
    double acc = 0.0;
    // (the loop bound is the same for the lanes of a row and rounded up to whole warps)
    const int64_t rows = ((int64_t)p.nfit + 32 / L - 1) / (32 / L) * (32 / L);
    for (int64_t i = t0 / L; i < rows; i += step / L) {
        const bool in = i < p.nfit;
        double yi = 0.0, vi = 0.0, ri = 0.0;
        if (in && sub == 0) {
            vi = p.v[i];
            if (upd) ri = p.r1[i];
            if (!ITEMS) yi = p.ba[i];
        }
        if (ITEMS) {
            double a0 = 0.0, a1 = 0.0, s0 = 0.0, s1 = 0.0;
            if (in) {
#pragma unroll 9
                for (int k = sub; k < C; k += L) a0 = fma(p.UWc[(int64_t)k * p.n + i], cs[k], a0);
                const int32_t g = p.p2g[i] - 1;
                const double *pt = p.part + (i - (p.aig[g] - 1));
                const int64_t q1 = p.itemBeg[g + 1];
                int64_t q = p.itemBeg[g] + sub;
                for (; q + 3 * L < q1; q += 4 * L) {
                    const double a = pt[q * p.R], b = pt[(q + L) * p.R], c = pt[(q + 2 * L) * p.R],
                                 d = pt[(q + 3 * L) * p.R];
                    s0 += a + b;
                    s1 += c + d;
                }
                for (; q < q1; q += L) a1 += pt[q * p.R];
            }
            yi = ((s0 + s1) + a1) - a0;
#pragma unroll
            for (int o = L / 2; o > 0; o >>= 1) yi += __shfl_xor_sync(0xffffffffu, yi, o);
        }
        if (in && sub == 0) {
            yi = yi - f * ri;
            p.y[i] = yi;
            acc += vi * yi;
        }
    }
    acc = cta_sum<kY1Threads>(acc, sh);
    if (threadIdx.x == 0) p.partA[blockIdx.x] = acc;
}

// alfa = v . y; the new residual r = y - (alfa / beta) r2 into the buffer of
// the one before r2; y = M^-1 r (diagonal cu), partials of r . y
__global__ void __launch_bounds__(kThreads) k_mr_y2(int32_t n, const MinresState *S, MinresFlags *F,
                                                    const double *partA, int npA, double *y, double *rOld,
                                                    const double *r2, const double *cu, double *partB) {
    __shared__ double sh[kThreads / 32], sf;
    if (F->done) return;
    if (threadIdx.x < 32) {
        const double alfa = warp_sum_of(partA, npA);
        if (threadIdx.x == 0) {
            sf = alfa * S->invb;
            if (blockIdx.x == 0) F->alfa = alfa;
        }
    }
    __syncthreads();
    const double f = sf;
    double acc = 0.0;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x) {
        const double yi = y[i] - f * r2[i];
        rOld[i] = yi;
        const double zi = (yi * cu[i]) * cu[i];
        y[i] = zi;
        acc += yi * zi;
    }
    acc = cta_sum<kThreads>(acc, sh);
    if (threadIdx.x == 0) partB[blockIdx.x] = acc;
}

// The scalar steps run in one warp on the CTA's copies; the square roots and
// reciprocals that do not depend on each other are taken by different lanes
// at once (a chain of them, 0.7 us each, was half of the kernel).
__device__ __forceinline__ double lane_of(double v, int lane) { return __shfl_sync(0xffffffffu, v, lane); }

// beta_{k+1} = sqrt(b2) and the left reflection
__device__ void mr_rotate(MinresState *S, double b2) {
    const int ln = threadIdx.x & 31;
    if (b2 < 0.0) {
        if (ln == 0) S->istop = 9;
        return;
    }
    const double gbar = S->sn * S->dbar - S->cs * S->alfa;
    double r = sqrt(ln == 0 ? b2 : gbar * gbar + b2);
    if (ln != 0 && r < 2.220446049250313e-16) r = 2.220446049250313e-16;
    const double inv = 1.0 / r;
    const double beta = lane_of(r, 0), invb = lane_of(inv, 0), gamma = lane_of(r, 1), denom = lane_of(inv, 1);
    if (ln) return;
    S->oldb = S->beta;
    S->beta = beta;
    S->bo = beta * S->invb;
    S->invb = invb;
    S->tnorm2 += S->alfa * S->alfa + S->oldb * S->oldb + b2;
    S->oldeps = S->epsln;
    S->delta = S->cs * S->dbar + S->sn * S->alfa;
    S->gbar = gbar;
    S->epsln = S->sn * beta;
    S->dbar = -S->cs * beta;
    S->cs = gbar * denom;
    S->sn = beta * denom;
    S->phi = S->cs * S->phibar;
    S->phibar = S->sn * S->phibar;
    S->denom = denom;
    S->gmax = fmax(S->gmax, gamma);
    S->gmin = fmin(S->gmin, gamma);
}

// beta_{k+1}, the left reflection (column k of R, tau_k), the right
// reflections P(k-2,k), P(k-1,k) and u: the oracle's steps, with products by
// reciprocals for its quotients
__device__ void qlp_rotate(MinresState *S, QlpState *Q, double b2) {
    const int ln = threadIdx.x & 31;
    if (b2 < 0.0) {
        if (ln == 0) S->istop = 9;
        return;
    }
    const int k = S->k + 1;
    const double epsk = S->epsln, alfa = S->alfa, oldb = S->beta;
    const double delta = S->cs * S->dbar + S->sn * alfa;
    const double gbar = S->sn * S->dbar - S->cs * alfa;
    const double tnorm2 = S->tnorm2 + (alfa * alfa + oldb * oldb + b2);
    // lanes: beta, gamma, the first right reflection, ||T||
    const double sq = ln == 0 ? b2 : ln == 1 ? gbar * gbar + b2 : ln == 2 ? Q->gA * Q->gA + epsk * epsk : tnorm2;
    const double rt = sqrt(sq), inv = rt > 0.0 ? 1.0 / rt : 0.0;
    const double beta = lane_of(rt, 0), invb = lane_of(inv, 0), gamma = lane_of(rt, 1), ig = lane_of(inv, 1);
    const double rA = lane_of(rt, 2), iA = lane_of(inv, 2), Anorm = lane_of(rt, 3);
    const double cs = gamma > 0.0 ? gbar * ig : 1.0, sn = gamma > 0.0 ? beta * ig : 0.0;
    const double tau = cs * S->phibar;
    double c1 = 1, s1 = 0, c2 = 1, s2 = 0, etaC = 0, thC = 0, gC, dk = delta, gk = gamma;
    double gA = Q->gA, thB = Q->thB, gB = Q->gB, iB = 0.0;
    if (k >= 3) {
        if (rA > 0.0) { c1 = gA * iA; s1 = epsk * iA; }
        gA = rA;
        const double th = c1 * thB + s1 * dk;
        dk = s1 * thB - c1 * dk;
        thB = th;
        etaC = s1 * gk;
        gk = -c1 * gk;
    }
    if (k >= 2) {
        const double r = sqrt(gB * gB + dk * dk);
        if (r > 0.0) { iB = 1.0 / r; c2 = gB * iB; s2 = dk * iB; }
        gB = r;
        thC = s2 * gk;
        gC = -c2 * gk;
    } else {
        gC = gk;
    }
    const double tiny = 2.220446049250313e-16 * Anorm;
    double uA = 0.0, uB = 0.0;
    if (k >= 3) uA = fabs(gA) > tiny ? (Q->tauA - Q->etaA * Q->uF2 - Q->thA * Q->uF1) * iA : 0.0;
    if (k >= 2) uB = fabs(gB) > tiny ? (Q->tauB - Q->etaB * Q->uF1 - thB * uA) * iB : 0.0;
    const double uC = fabs(gC) > tiny ? (tau - etaC * uA - thC * uB) / gC : 0.0;
    __syncwarp();
    if (ln) return;
    S->oldb = oldb;
    S->beta = beta;
    S->bo = beta * S->invb;
    S->invb = invb;
    S->tnorm2 = tnorm2;
    S->Anorm = Anorm;
    S->gbar = gbar;
    S->epsln = S->sn * beta;
    S->dbar = -S->cs * beta;
    S->cs = cs;
    S->sn = sn;
    S->phibar = sn * S->phibar;
    S->gmax = fmax(S->gmax, gamma);
    S->gmin = fmin(S->gmin, gamma);
    Q->c1 = c1; Q->s1 = s1; Q->c2 = c2; Q->s2 = s2;
    Q->uA = uA; Q->uB = uB; Q->uC = uC;
    if (k >= 3) { Q->uF2 = Q->uF1; Q->uF1 = uA; }
    Q->etaA = Q->etaB; Q->thA = thB; Q->gA = gB; Q->tauA = Q->tauB;
    Q->etaB = etaC; Q->thB = thC; Q->gB = gC; Q->tauB = tau;
}

// The scalar step from beta^2 = r . y (in every CTA), the solution update
// with the current Lanczos vector v (MINRES: w into the buffer of the older
// of the two kept, x; MINRES-QLP: W = V P with w_{k-2} final into xp, and
// the candidate iterate xc), partials of x . x; then the next vector v = y /
// beta, padded with zeros for the operator (xa), and the partial dots of it
// with the 2 m columns [U | W] of the constraint reflections (row-major
// UWr: a thread owns a column and every nsub-th row, so that no sum crosses
// lanes but the last nsub ones; 36 columns of 30,000 rows are 1.7 us of
// FP64).  kStart: the first vector only.
enum StepKind { kStart, kMinres, kQlp };

struct StepParams {
    int32_t n, nfit, m, R;
    const int32_t *aig, *p2g;   // padded positions of xa (aig null: xa has the order of the parameters)
    const MinresState *Sin;
    MinresState *Sout;
    const QlpState *Qin;
    QlpState *Qout;
    const MinresFlags *F;
    const double *partB;
    int npB;
    const double *y, *UWr;
    double *v, *xa, *partX, *partUW;
    double *wa, *wb, *x, *xp, *xc;   // MINRES: wa the older, wb the newer w
};

template <StepKind KIND>
__global__ void __launch_bounds__(kThreads) k_mr_step(StepParams p) {
    __shared__ double sh[kThreads / 32], xs[kStepRows], red[kThreads];
    __shared__ MinresState ss;
    __shared__ QlpState qs;
    if (p.F->done) return;
    const int tid = threadIdx.x;
    // the CTA's copies of the scalars, by words
    if (tid < (int)(sizeof(MinresState) / 8))
        reinterpret_cast<double *>(&ss)[tid] = reinterpret_cast<const double *>(p.Sin)[tid];
    if (KIND == kQlp && tid >= 32 && tid < 32 + (int)(sizeof(QlpState) / 8))
        reinterpret_cast<double *>(&qs)[tid - 32] = reinterpret_cast<const double *>(p.Qin)[tid - 32];
    __syncthreads();
    if (KIND != kStart && tid < 32) {
        const double b2 = warp_sum_of(p.partB, p.npB);
        if (tid == 0) ss.alfa = p.F->alfa;
        __syncwarp();
        if (KIND == kQlp) qlp_rotate(&ss, &qs, b2);
        else mr_rotate(&ss, b2);
        if (tid == 0) {
            ss.k += 1;
            if (blockIdx.x == 0) {
                *p.Sout = ss;
                if (KIND == kQlp) *p.Qout = qs;
            }
        }
    }
    __syncthreads();
    if (ss.istop == 9) return;
    const int k = ss.k;
    const double f = ss.invb;
    const int C = 2 * p.m;
    const int nsub = C ? kThreads / C : 0, sub = C ? tid / C : 0, cc = C ? tid - sub * C : 0;
    double acc = 0.0, xx = 0.0;
    for (int64_t r0 = (int64_t)blockIdx.x * kStepRows; r0 < p.n; r0 += (int64_t)gridDim.x * kStepRows) {
        const int64_t i = r0 + tid;
        if (tid < kStepRows) {
            double vi = 0.0;
            if (i < p.nfit) {
                if (KIND == kMinres) {
                    const double wn = (p.v[i] - ss.oldeps * p.wa[i] - ss.delta * p.wb[i]) * ss.denom;
                    p.wa[i] = wn;
                    const double xi = p.x[i] + ss.phi * wn;
                    p.x[i] = xi;
                    xx += xi * xi;
                } else if (KIND == kQlp) {
                    double a = p.wa[i], bb = p.wb[i], c = p.v[i], xi = p.xp[i];
                    if (k >= 3) {
                        const double a2 = qs.c1 * a + qs.s1 * c;
                        c = qs.s1 * a - qs.c1 * c;
                        a = a2;
                        xi = xi + qs.uA * a;
                        p.xp[i] = xi;
                    }
                    if (k >= 2) {
                        const double b2r = qs.c2 * bb + qs.s2 * c;
                        c = qs.s2 * bb - qs.c2 * c;
                        bb = b2r;
                    }
                    p.wa[i] = bb;
                    p.wb[i] = c;
                    xi = xi + qs.uB * bb + qs.uC * c;
                    p.xc[i] = xi;
                    xx += xi * xi;
                }
                vi = f * p.y[i];
                p.v[i] = vi;
            }
            if (i < p.n) {
                int64_t at = i;
                if (p.aig) {
                    const int32_t g = p.p2g[i] - 1;
                    at = (int64_t)g * p.R + i - (p.aig[g] - 1);
                }
                p.xa[at] = vi;
            }
            xs[tid] = vi;
        }
        if (!C) continue;
        __syncthreads();
        if (sub < nsub) {
            const int rows = (int)min((int64_t)kStepRows, p.n - r0);
            const double *u = p.UWr + r0 * C + cc;
#pragma unroll 10
            for (int r = sub; r < rows; r += nsub) acc = fma(u[(int64_t)r * C], xs[r], acc);
        }
        __syncthreads();
    }
    if (KIND != kStart) {
        xx = cta_sum<kThreads>(xx, sh);
        if (tid == 0) p.partX[blockIdx.x] = xx;
    }
    if (!C) return;
    red[tid] = acc;
    __syncthreads();
    if (tid < C) {
        double t = 0.0;
        for (int q = 0; q < nsub; ++q) t += red[q * C + tid];
        p.partUW[(int64_t)blockIdx.x * C + tid] = t;
    }
}

__global__ void k_apply_precond(int32_t n, const double *r, const double *cu, double *y) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        y[i] = (r[i] * cu[i]) * cu[i];
}

// ---- the reflections as columns: U (n x m, column k = V_k with Vk at n - m + k)
__global__ void k_u_columns(int32_t n, int32_t m, const double *V, const double *Vk, double *U) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < (int64_t)n * m;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = e / n, i = e - k * n, kn = n - m + k;
        U[e] = i < kn ? V[e] : (i == kn ? Vk[k] : 0.0);
    }
}

// M = U^T W, one CTA per element
__global__ void __launch_bounds__(kThreads) k_column_dots(int32_t n, int32_t m, const double *U, const double *W,
                                                          double *M) {
    __shared__ double sh[kThreads / 32];
    const double *u = U + (int64_t)(blockIdx.x / m) * n, *w = W + (int64_t)(blockIdx.x % m) * n;
    double v = 0.0;
    for (int i = threadIdx.x; i < n; i += kThreads) v = fma(u[i], w[i], v);
    v = cta_sum<kThreads>(v, sh);
    if (threadIdx.x == 0) M[blockIdx.x] = v;
}

// S = T M T^T (T upper triangular), one CTA; X scratch
__global__ void k_wy_s(int32_t m, const double *T, const double *M, double *X, double *S) {
    for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
        const int r = e / m, c = e % m;
        double v = 0.0;
        for (int q = r; q < m; ++q) v = fma(T[r * m + q], M[q * m + c], v);
        X[e] = v;
    }
    __syncthreads();
    for (int e = threadIdx.x; e < m * m; e += blockDim.x) {
        const int r = e / m, c = e % m;
        double v = 0.0;
        for (int q = c; q < m; ++q) v = fma(X[r * m + q], T[c * m + q], v);
        S[e] = v;
    }
}

// Z = W T^T - U S / 2, so that Q^T A Q = A - Z U^T - U Z^T; [U | W] by rows
__global__ void k_wy_zrows(int32_t n, int32_t m, const double *U, const double *W, const double *T, const double *S,
                           double *Z, double *UWr) {
    for (int64_t e = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; e < (int64_t)n * m;
         e += (int64_t)gridDim.x * blockDim.x) {
        const int64_t k = e / n, i = e - k * n;
        double z = 0.0, h = 0.0;
        for (int64_t b = k; b < m; ++b) z = fma(W[b * n + i], T[k * m + b], z);
        for (int64_t b = 0; b < m; ++b) h = fma(U[b * n + i], S[b * m + k], h);
        Z[e] = z - 0.5 * h;
        UWr[i * 2 * m + k] = U[e];
        UWr[i * 2 * m + m + k] = W[e];
    }
}

// diagonal of Q^T A Q
__global__ void k_diag_eliminate(int32_t n, int32_t m, const double *U, const double *Z, double *dg) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    double a = 0.0;
    for (int64_t k = 0; k < m; ++k) a = fma(Z[k * n + i], U[k * n + i], a);
    dg[i] = dg[i] - 2.0 * a;
}

__global__ void k_precond(int32_t n, const double *dg, double *cu) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        cu[i] = dg[i] > 0.0 ? 1.0 / sqrt(dg[i]) : 0.0;
}

__global__ void k_diag_update(int32_t n, double *dg, const double *v, const double *y, const double *betap) {
    const double beta = *betap;
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dg[i] = dg[i] - 4.0 * v[i] * y[i] + 4.0 * beta * v[i] * v[i];
}

__global__ void k_sparse_diag(int32_t n, const double *matD, double *dg) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        dg[i] = matD[i];
}

__global__ void k_fill(int32_t n, double v, double *a) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        a[i] = v;
}

__global__ void k_sub(int32_t n, double *a, const double *b) {
    for (int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x; i < n; i += (int64_t)gridDim.x * blockDim.x)
        a[i] = a[i] - b[i];
}

// ---------------------------------------------------------------- helpers
// device memory that a context keeps between its iterative solves, at most, for
// the block-row copy and for the vectors each (30,000 globals: 145 and 70 MB)
constexpr int64_t kKeepBytes = (int64_t)4 << 30;

struct Solver {
    mpgpu_ctx *c;
    DevJob &j;
    cudaStream_t s;
    int nsm;
    SparseBlocks sb;
    bool useRows = false;         // the product takes the job's block-row copy
    double *part = nullptr, *partOwned = nullptr;   // partial sums of dot()
    explicit Solver(mpgpu_ctx *cc) : c(cc), j(cc->j), s(cc->stream) {
        cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device);
    }
    ~Solver() {
        // the copy and the vectors stay for the next solve unless they are large:
        // the data loop in between may need the memory
        if (useRows && block_rows_bytes(j.br) > kKeepBytes) block_rows_free(j);
        if (8 * j.cap[(const void *)&j.work] > kKeepBytes) dfree(j.work);
        // stream-ordered (cudaMallocAsync on the context's stream)
        if (partOwned) cudaFreeAsync(partOwned, s);
        dfree(wyPart); dfree(wyT);
        dfree(sb.rowStart); dfree(sb.bcol); dfree(sb.boff); dfree(sb.bld); dfree(sb.tOff);
        dfree(sb.colStart); dfree(sb.colBlk); dfree(sb.tBase); dfree(sb.tbuf);
        dfree(sb.tStr); dfree(sb.brow); dfree(sb.rowPart);
        dfree(sb.colItemJ); dfree(sb.colItemQ0); dfree(sb.colItemQ1); dfree(sb.colItemBeg); dfree(sb.colPart);
        dfree(pmvRow); dfree(pmvPart);
    }
    unsigned grid(int64_t n, int per = kThreads) const {
        int64_t g = (n + per - 1) / per;
        int64_t m = (int64_t)nsm * 8;
        if (g > m) g = m;
        return (unsigned)(g < 1 ? 1 : g);
    }
    unsigned wgrid(int64_t nwarp) const { return grid(nwarp * 32); }

    // packed symmetric product (two passes; buffers kept for the solve)
    double *pmvRow = nullptr, *pmvPart = nullptr;
    int64_t pmvN = 0;
    // scratch of the packed product; a failed allocation leaves none (the
    // product is then not launched and pmvFailed is set)
    cudaError_t alloc_pmv(int32_t n) {
        if (pmvN == n && pmvRow && pmvPart) return cudaSuccess;
        const int64_t nb = ((int64_t)n + kMvRows - 1) / kMvRows;
        dfree(pmvRow);
        dfree(pmvPart);
        pmvN = -1;
        const int64_t nch = ((int64_t)n + kMvCols - 1) / kMvCols;
        cudaError_t e = cudaMalloc(&pmvRow, sizeof(double) * std::max<int64_t>(nch * n, 1));
        if (e == cudaSuccess) e = cudaMalloc(&pmvPart, sizeof(double) * std::max<int64_t>(nb * n, 1));
        if (e != cudaSuccess) {
            dfree(pmvRow);
            dfree(pmvPart);
            pmvFailed = true;
            return e;
        }
        pmvN = n;
        return cudaSuccess;
    }
    bool pmvFailed = false;
    void packed_matvec(int32_t n, const double *A, const double *x, double *y) {
        const int64_t nb = ((int64_t)n + kMvRows - 1) / kMvRows;
        if (alloc_pmv(n) != cudaSuccess) return;
        const dim3 grid((unsigned)nb, (unsigned)(((int64_t)n + kMvCols - 1) / kMvCols));
        k_pmv_blocks<<<grid, 256, 0, s>>>(n, A, x, pmvRow, pmvPart);
        k_pmv_final<<<(unsigned)((n + 31) / 32), 256, 0, s>>>(n, nb, pmvRow, pmvPart, y);
    }

    // block table of the sparse storage, built from the host copies
    int32_t build_blocks() {
        std::vector<int64_t> off(2 * (j.nG + 1));
        std::vector<int32_t> col(std::max<int64_t>(j.ncolw, 1));
        cudaMemcpy(off.data(), j.off, sizeof(int64_t) * off.size(), cudaMemcpyDeviceToHost);
        if (j.ncolw > 0) cudaMemcpy(col.data(), j.col, sizeof(int32_t) * j.ncolw, cudaMemcpyDeviceToHost);
        const std::vector<int32_t> &aig = j.hAig;
        std::vector<int64_t> rowStart(1, 0), boff, tOff;
        std::vector<int32_t> bcol, bld;
        int64_t tl = 0;
        for (int32_t I = 1; I <= j.nG; ++I) {
            const int32_t np = aig[I] - aig[I - 1];
            const int64_t kk = off[2 * (I - 1)], ll = off[2 * (I - 1) + 1];
            const int64_t ku = off[2 * I] - kk;
            if (ku > 0) {
                if (col[kk] != 0) {  // uncompressed: one (np x ku) matrix
                    int64_t k = 0;
                    while (k < ku) {
                        const int32_t first = col[kk + k];
                        // group of this column
                        int32_t J = (int32_t)(std::upper_bound(aig.begin(), aig.end(), first) - aig.begin());
                        const int32_t nj = aig[J] - aig[J - 1];
                        bcol.push_back(J);
                        boff.push_back(ll + k);
                        bld.push_back((int32_t)ku);
                        tOff.push_back(J == I ? -1 : tl);
                        if (J != I) tl += nj;
                        k += nj;
                    }
                } else {  // compressed: regions (offset, first group) ... (end offset, n+1)
                    for (int64_t k = 2; k <= ku - 2; k += 2) {
                        const int32_t g0 = col[kk + k - 1];
                        const int32_t o0 = col[kk + k - 2];
                        const int32_t o1 = col[kk + k];
                        const int32_t width = o1 - o0;
                        int32_t inreg = 0, J = g0;
                        while (inreg < width) {
                            const int32_t nj = aig[J] - aig[J - 1];
                            bcol.push_back(J);
                            boff.push_back(ll + (int64_t)o0 * np + inreg);
                            bld.push_back(width);
                            tOff.push_back(J == I ? -1 : tl);
                            if (J != I) tl += nj;
                            inreg += nj;
                            J++;
                        }
                    }
                }
            }
            rowStart.push_back((int64_t)bcol.size());
        }
        // incoming (transposed) blocks per column group, ordered by row group
        const int64_t nb = (int64_t)bcol.size();
        std::vector<int64_t> cnt(j.nG + 2, 0);
        std::vector<int32_t> brow(nb);
        for (int32_t I = 1; I <= j.nG; ++I)
            for (int64_t b = rowStart[I - 1]; b < rowStart[I]; ++b) brow[b] = I;
        for (int64_t b = 0; b < nb; ++b)
            if (bcol[b] != brow[b]) cnt[bcol[b]]++;
        std::vector<int64_t> colStart(j.nG + 1, 0);
        for (int32_t J = 1; J <= j.nG; ++J) colStart[J] = colStart[J - 1] + cnt[J];
        std::vector<int64_t> fill(colStart.begin(), colStart.end() - 1), colBlk(std::max<int64_t>(colStart[j.nG], 1));
        for (int64_t b = 0; b < nb; ++b)
            if (bcol[b] != brow[b]) colBlk[fill[bcol[b] - 1]++] = b;
        int32_t maxnp = 0;
        for (int32_t I = 1; I <= j.nG; ++I) maxnp = std::max(maxnp, aig[I] - aig[I - 1]);
        sb.smallGroups = maxnp <= kSmallGroup && nb < (int64_t)0xffffffff;
        // transposed products stored by column group, incoming blocks in row
        // group order: block after block (general kernels) or parameter-major
        // with the group's block count as stride (small groups)
        std::vector<int64_t> tBase(std::max(j.nG, 1));
        std::vector<int32_t> tStr(std::max<int64_t>(nb, 1), 1);
        {
            int64_t off = 0;
            for (int32_t J = 1; J <= j.nG; ++J) {
                tBase[J - 1] = off;
                const int32_t nj = aig[J] - aig[J - 1];
                const int64_t cnt = colStart[J] - colStart[J - 1];
                for (int64_t q = colStart[J - 1]; q < colStart[J]; ++q) {
                    const int64_t r = q - colStart[J - 1];
                    tOff[colBlk[q]] = sb.smallGroups ? off + r : off + r * nj;
                    tStr[colBlk[q]] = (int32_t)cnt;
                }
                off += cnt * nj;
            }
        }
        std::vector<int32_t> ciJ;
        std::vector<int64_t> ciQ0, ciQ1, ciBeg(j.nG + 1, 0);
        for (int32_t J = 1; J <= j.nG; ++J) {
            ciBeg[J - 1] = (int64_t)ciJ.size();
            const int64_t cnt = colStart[J] - colStart[J - 1];
            int64_t q = 0;
            do {
                ciJ.push_back(J);
                ciQ0.push_back(q);
                ciQ1.push_back(std::min<int64_t>(cnt, q + kColItem));
                q += kColItem;
            } while (q < cnt);
        }
        ciBeg[j.nG] = (int64_t)ciJ.size();
        sb.nColItem = (int64_t)ciJ.size();
        int32_t minnp = maxnp;
        for (int32_t I = 1; I <= j.nG; ++I) minnp = std::min(minnp, aig[I] - aig[I - 1]);
        sb.uniform = (sb.smallGroups && minnp == maxnp) ? maxnp : 0;
        sb.nblk = nb;
        sb.tlen = tl;
        auto up = [&](auto *&d, const auto &h) -> cudaError_t {
            cudaError_t e = cudaMalloc((void **)&d, sizeof(h[0]) * std::max<size_t>(h.size(), 1));
            if (e != cudaSuccess) return e;
            return cudaMemcpy(d, h.data(), sizeof(h[0]) * h.size(), cudaMemcpyHostToDevice);
        };
        MPG_CUDA(c, up(sb.rowStart, rowStart));
        MPG_CUDA(c, up(sb.bcol, bcol));
        MPG_CUDA(c, up(sb.boff, boff));
        MPG_CUDA(c, up(sb.bld, bld));
        MPG_CUDA(c, up(sb.tOff, tOff));
        MPG_CUDA(c, up(sb.colStart, colStart));
        MPG_CUDA(c, up(sb.colBlk, colBlk));
        MPG_CUDA(c, up(sb.tBase, tBase));
        if (sb.smallGroups) {
            MPG_CUDA(c, up(sb.tStr, tStr));
            MPG_CUDA(c, up(sb.brow, brow));
            MPG_CUDA(c, cudaMalloc((void **)&sb.rowPart, sizeof(double) * std::max<int64_t>(nb, 1) * kSmallGroup));
            MPG_CUDA(c, up(sb.colItemJ, ciJ));
            MPG_CUDA(c, up(sb.colItemQ0, ciQ0));
            MPG_CUDA(c, up(sb.colItemQ1, ciQ1));
            MPG_CUDA(c, up(sb.colItemBeg, ciBeg));
            MPG_CUDA(c, cudaMalloc((void **)&sb.colPart, sizeof(double) * std::max<int64_t>(sb.nColItem, 1) * kSmallGroup));
        }
        MPG_CUDA(c, cudaMalloc((void **)&sb.tbuf, sizeof(double) * std::max<int64_t>(tl, 1)));
        return MPGPU_OK;
    }

    // what avprd0 needs for the current matrix
    int32_t prepare_product() {
        if (j.matsto != 2) {
            MPG_CUDA(c, alloc_pmv(j.nVar));
            return MPGPU_OK;
        }
        useRows = !c->lean && block_rows_fit(c);
        if (useRows && block_rows_build(c) == MPGPU_OK) return MPGPU_OK;
        return from_storage();
    }

    // the product from the stored matrix: layouts that the copy does not
    // serve, or no memory for it (the copy takes twice the matrix, the
    // transposed products 0.4 of it for groups of six)
    int32_t from_storage() {
        if (useRows) {
            cudaGetLastError();
            block_rows_free(j);
        }
        useRows = false;
        return build_blocks();
    }

    // y = A x (full parameter space)
    void avprd0(const double *x, double *y) {
        if (useRows) {
            block_rows_product(j.br, j.aig, j.p2g, x, y, s);
        } else if (j.matsto == 2 && sb.smallGroups) {
            const unsigned gb = grid(sb.nblk);
            auto blocks = [&](auto g) {
                k_spmv_blocks<decltype(g)::value><<<gb, kThreads, 0, s>>>(sb.nblk, sb.brow, j.aig, sb.bcol, sb.boff, sb.bld,
                                                                          sb.tOff, sb.tStr, j.matD, x, sb.tbuf,
                                                                          sb.rowPart);
            };
            switch (sb.uniform) {
            case 1: blocks(std::integral_constant<int, 1>()); break;
            case 2: blocks(std::integral_constant<int, 2>()); break;
            case 3: blocks(std::integral_constant<int, 3>()); break;
            case 4: blocks(std::integral_constant<int, 4>()); break;
            case 5: blocks(std::integral_constant<int, 5>()); break;
            case 6: blocks(std::integral_constant<int, 6>()); break;
            case 7: blocks(std::integral_constant<int, 7>()); break;
            case 8: blocks(std::integral_constant<int, 8>()); break;
            default: blocks(std::integral_constant<int, 0>()); break;
            }
            k_spmv_colitems<<<wgrid(sb.nColItem), kThreads, 0, s>>>(sb.nColItem, sb.colItemJ, sb.colItemQ0,
                                                                    sb.colItemQ1, j.aig, sb.rowStart, sb.rowPart,
                                                                    sb.colStart, sb.tBase, sb.tbuf, sb.colPart);
            k_spmv_final<<<grid(j.nVar), kThreads, 0, s>>>(j.nVar, j.aig, j.p2g, sb.colItemBeg, sb.colPart, j.matD,
                                                           x, y);
        } else if (j.matsto == 2) {
            k_spmv_rows<<<wgrid(j.nG), kThreads, 0, s>>>(j.nG, j.aig, sb.rowStart, sb.bcol, sb.boff, sb.bld,
                                                         sb.tOff, j.matD, x, y, sb.tbuf);
            k_spmv_cols<<<wgrid(j.nG), kThreads, 0, s>>>(j.nG, j.aig, sb.colStart, sb.colBlk, sb.tOff,
                                                         sb.tbuf, y);
        } else {
            packed_matvec(j.nVar, j.matD, x, y);
        }
    }
    // the reflections of qlssq in its order (k = m..1): v = v_k, yk =
    // P^T A P v_k with P = H_m ... H_{k+1}, *dsc = v.yk; apply() after each
    template <class Fn>
    void reflections(double *v, double *tmp, double *yk, double *dsc, Fn &&apply) {
        const int32_t n = j.nVar, ncon = j.ncon;
        for (int k = ncon; k >= 1; --k) {
            const int kn = n + k - ncon;
            const double *vr = j.qlV + (int64_t)(k - 1) * n;
            k_vec_with_kn<<<grid(n), kThreads, 0, s>>>(vr, j.hR2[k - 1], j.hVk[k - 1], kn, n, v);
            cudaMemcpyAsync(tmp, v, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
            if (k < ncon) k_qlapply<<<1, 1024, 0, s>>>(tmp, j.qlV, j.qlVk, j.qlR2, n, ncon, k + 1, ncon, 1);
            avprd0(tmp, yk);
            if (k < ncon) k_qlapply<<<1, 1024, 0, s>>>(yk, j.qlV, j.qlVk, j.qlR2, n, ncon, ncon, k + 1, -1);
            dot(v, yk, n, part, dsc, s);
            apply();
        }
    }
    // Reflections of at most kWyFused constraints as n x m columns: U, W = A
    // U, Z with Q^T A Q = A - Z U^T - U Z^T (its diagonal and band follow
    // without applying reflection after reflection), S = T (U^T A U) T^T, and
    // [U | W] by rows for the iteration's dot products.  Q^T A Q x = A x - W a
    // - U c with a = T^T s, c = T t - S s, s = U^T x, t = W^T x: the 2 m dots
    // and one product with the unreflected x, instead of a reflection pass
    // before and after the product.
    struct Wy {
        int32_t m = 0;
        double *UWc = nullptr, *UWr = nullptr, *Z = nullptr, *S = nullptr;
    } wy;
    bool wy_fits() const { return useRows && j.ncon > 0 && j.ncon <= kWyFused; }
    int64_t wy_len() const { return wy_fits() ? 5 * (int64_t)j.ncon * j.nVar + 3 * (int64_t)j.ncon * j.ncon : 0; }
    // buf: wy_len() doubles
    int32_t wy_build(double *buf) {
        const int32_t m = j.ncon, n = j.nVar;
        const int64_t nm = (int64_t)n * m;
        wy.UWc = buf;
        wy.UWr = buf + 2 * nm;
        wy.Z = buf + 4 * nm;
        wy.S = buf + 5 * nm;
        double *M = wy.S + m * m, *X = M + m * m;
        k_u_columns<<<grid(nm), kThreads, 0, s>>>(n, m, j.qlV, j.qlVk, wy.UWc);
        for (int32_t k = 0; k < m; ++k)
            MPG_CUDA(c, block_rows_product(j.br, j.aig, j.p2g, wy.UWc + (int64_t)k * n, wy.UWc + nm + (int64_t)k * n, s));
        k_column_dots<<<m * m, kThreads, 0, s>>>(n, m, wy.UWc, wy.UWc + nm, M);
        k_wy_s<<<1, 1024, 0, s>>>(m, j.qlT, M, X, wy.S);
        k_wy_zrows<<<grid(nm), kThreads, 0, s>>>(n, m, wy.UWc, wy.UWc + nm, j.qlT, wy.S, wy.Z, wy.UWr);
        MPG_CUDA(c, cudaGetLastError());
        wy.m = m;
        return MPGPU_OK;
    }

    // band of Q^T A Q (pede's preconditioner fill and qlpssq with band
    // width mbandw) and its lltdec factor with the block spikes
    int32_t band_build(BandPre &P, int32_t mbandw, int32_t lprecm, double *v, double *tmp, double *yk,
                       double *dsc) {
        const int32_t n = j.nVar, nfit = j.nVar - j.ncon;
        if (mbandw > MPGPU_BAND_MAX) return set_err(c, MPGPU_ERR_LIMIT, "band preconditioner wider than 32");
        if (band_alloc(P, n, nfit, mbandw - 1)) return set_err(c, MPGPU_ERR_ALLOC, "band preconditioner");
        MPG_CUDA(c, band_fill(P, n, j.matsto, j.matD, j.aig, j.p2g, j.rowBlk0, j.blkJ, j.blkOff, j.blkLd, j.nmat, s));
        if (wy.m > 0) {
            MPG_CUDA(c, band_eliminate(P, n, wy.m, wy.UWc, wy.Z, s));
        } else {
            cudaError_t e = cudaSuccess;
            reflections(v, tmp, yk, dsc, [&] {
                if (e == cudaSuccess) e = band_reflect(P, n, v, yk, dsc, s);
            });
            MPG_CUDA(c, e);
        }
        MPG_CUDA(c, band_factor(P, lprecm, s));
        return MPGPU_OK;
    }
    // qlmlq (mpqldec.f90:404-454): t = 1 Q^T x (reflections ncon..1), t = 0
    // Q x (1..ncon), in the compact WY form
    double *wyPart = nullptr, *wyT = nullptr;
    void qlmlq(double *x, int t) {
        if (j.ncon <= 0) return;
        const int32_t m = j.ncon, n = j.nVar;
        if (!wyPart && m <= 4096) {
            if (cudaMalloc(&wyPart, sizeof(double) * (size_t)kWyBlocks * m) != cudaSuccess ||
                cudaMalloc(&wyT, sizeof(double) * m) != cudaSuccess) {
                dfree(wyPart);
                dfree(wyT);
                cudaGetLastError();
            }
        }
        // coefficients beyond the shared memory of one CTA, or no workspace:
        // the reflections one after the other in one CTA
        if (m > 4096 || !wyPart || !wyT) {
            if (t) k_qlapply<<<1, 1024, 0, s>>>(x, j.qlV, j.qlVk, j.qlR2, n, m, m, 1, -1);
            else k_qlapply<<<1, 1024, 0, s>>>(x, j.qlV, j.qlVk, j.qlR2, n, m, 1, m, 1);
            return;
        }
        const int nb = (int)std::min<int64_t>(kWyBlocks, std::max<int64_t>(1, n / 512));
        k_wy_dots<<<nb, 256, 0, s>>>(n, m, j.qlV, x, wyPart);
        k_wy_coef<<<1, 256, sizeof(double) * m, s>>>(n, m, nb, wyPart, j.qlVk, j.qlT, x, t ? 0 : 1, wyT);
        k_wy_apply<<<grid(n), kThreads, sizeof(double) * m, s>>>(n, m, j.qlV, j.qlVk, wyT, x);
    }
};

}  // namespace

// ---------------------------------------------------------------- inversion / Cholesky
// minver / mchdec (pede.f90:7838-8054) on the packed matrix
int32_t solve_inversion(mpgpu_ctx *c, const double *consResiduals, double *corrOut, double *errs,
                        mpgpu_solveinfo *info, bool decomposition, int dense, double rtol, int32_t itnlim) {
    Solver S(c);
    DevJob &j = c->j;
    cudaStream_t s = c->stream;
    const int32_t n = j.nVar, ncon = j.ncon, nfit = n - ncon;
    if (j.matsto != 2 && ncon > 0) MPG_CUDA(c, S.alloc_pmv(n));   // the packed products of qlssq
    // per-solve vectors from the stream-ordered pool: a cudaFree would wait
    // for the whole device, i.e. for the other jobs' work in a served mix
    struct Tmp {
        cudaStream_t s;
        double *corr = nullptr, *vbuf = nullptr, *Av = nullptr, *work = nullptr, *diag = nullptr, *yv = nullptr;
        int32_t *used = nullptr, *piv = nullptr;
        ~Tmp() {
            for (void *p : {(void *)corr, (void *)vbuf, (void *)Av, (void *)work, (void *)diag, (void *)yv,
                            (void *)used, (void *)piv})
                if (p) cudaFreeAsync(p, s);
        }
    } T{s};
    double *&corr = T.corr, *&vbuf = T.vbuf, *&Av = T.Av, *&work = T.work, *&diag = T.diag, *&yv = T.yv;
    int32_t *&used = T.used, *&piv = T.piv;
    MPG_CUDA(c, cudaMallocAsync(&corr, sizeof(double) * n, s));
    MPG_CUDA(c, cudaMallocAsync(&vbuf, sizeof(double) * n, s));
    MPG_CUDA(c, cudaMallocAsync(&Av, sizeof(double) * n, s));
    if (dense < 0) MPG_CUDA(c, cudaMallocAsync(&work, sizeof(double) * packed_work_len(nfit), s));
    MPG_CUDA(c, cudaMallocAsync(&diag, sizeof(double) * n, s));
    MPG_CUDA(c, cudaMallocAsync(&yv, sizeof(double) * (ncon + 1), s));
    MPG_CUDA(c, cudaMallocAsync(&used, sizeof(int32_t) * n, s));
    MPG_CUDA(c, cudaMallocAsync(&piv, sizeof(int32_t) * 4, s));
    MPG_CUDA(c, cudaMallocAsync(&S.partOwned, sizeof(double) * (kDotBlocks + 8), s));
    S.part = S.partOwned;
    cudaEvent_t e0, e1;
    cudaEventCreate(&e0);
    cudaEventCreate(&e1);
    cudaEventRecord(e0, s);
    MPG_CUDA(c, cudaMemcpyAsync(corr, j.gvec, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    double *scal = c->scal + 300;   // device scalars
    // Q^T A Q (qlssq, reflections k = ncon .. 1)
    auto qlssq = [&](int t) {
        for (int jj = 1; jj <= ncon; ++jj) {
            const int k = t ? ncon + 1 - jj : jj;
            const int kn = n + k - ncon;
            const int ilast = j.hR2[k - 1];
            const double vkv = j.hVk[k - 1];
            const double *v = j.qlV + (int64_t)(k - 1) * n;
            k_vec_with_kn<<<S.grid(n), kThreads, 0, s>>>(v, ilast, vkv, kn, n, vbuf);
            S.avprd0(vbuf, Av);
            dot(vbuf, Av, n, S.part, scal, s);   // vtAv
            const dim3 tiles((unsigned)((n + kQlRows - 1) / kQlRows), (unsigned)((n + kQlCols - 1) / kQlCols));
            k_qlssq_update<<<tiles, 256, 0, s>>>(n, j.matD, v, vkv, Av, scal, ilast, kn);
        }
    };
    // tensor-core forms with up to 128 constraints: Q^T A Q is formed inside
    // the dense solve for the preconditioner only (compact WY, 3xTF32) and
    // the refinement applies Q in FP64; no FP64 sweep of the matrix here
    const bool wyElim = dense == 1 && ncon >= 1 && ncon <= 128;
    std::vector<double> y(ncon > 0 ? ncon : 1, 0.0);
    if (ncon > 0) {
        if (!wyElim) qlssq(1);
        // qlbsub (mpqldec.f90:991-1014) on the host
        for (int k = ncon; k >= 1; --k) {
            double d = 0.0;
            for (int cc = 1; cc <= ncon - k; ++cc) d = d + j.hL[(size_t)(k - 1) * ncon + k - 1 + cc] * y[k - 1 + cc];
            y[k - 1] = ((consResiduals ? consResiduals[k - 1] : 0.0) - d) / j.hL[(size_t)(k - 1) * ncon + k - 1];
        }
        MPG_CUDA(c, cudaMemcpyAsync(yv, y.data(), sizeof(double) * ncon, cudaMemcpyHostToDevice, s));
        if (!wyElim) {
            S.qlmlq(corr, 1);
            k_cons_rhs<<<S.grid(nfit), kThreads, 0, s>>>(nfit, ncon, j.matD, yv, corr);
        }
    }
    if (S.pmvFailed) return set_err(c, MPGPU_ERR_ALLOC, "packed product scratch");
    int nrank = 0;
    if (!decomposition && dense < 0) {
        // sqminl (mpnum.f90:230-355) on the leading nfit x nfit block
        k_diag_abs<<<S.grid(nfit), kThreads, 0, s>>>(nfit, j.matD, diag);
        MPG_CUDA(c, packed_sqminl(nfit, j.matD, corr, diag, used, piv, work, s));
        k_sqminl_deficit<<<S.grid(nfit, 1), kThreads, 0, s>>>(nfit, j.matD, corr, used, piv);
        k_negate<<<S.grid((int64_t)nfit * (nfit + 1) / 2), kThreads, 0, s>>>((int64_t)nfit * (nfit + 1) / 2, j.matD);
        std::vector<int32_t> hu(nfit);
        MPG_CUDA(c, cudaMemcpyAsync(hu.data(), used, sizeof(int32_t) * nfit, cudaMemcpyDeviceToHost, s));
        MPG_CUDA(c, cudaStreamSynchronize(s));
        for (int32_t u : hu) nrank += u;
    } else if (dense >= 0) {
        // blocked dense Cholesky (FP64, or tensor-core 3xTF32) refined by
        // preconditioned CG in FP64
        // (inversion forms: the inverse from the same factor replaces the
        // leading block of the packed matrix, where sqminl leaves it)
        const double tol = rtol > 0.0 ? rtol : 1e-13;
        const DenseWyElim wye{ncon, j.qlV, j.qlVk, j.qlT, yv};
        const int32_t rcd = wyElim ? dense_solve_pcg(c, n, j.matD, corr, dense, tol, itnlim > 0 ? itnlim : 2000,
                                                     info, decomposition ? nullptr : j.matD, &wye)
                                   : dense_solve_pcg(c, nfit, j.matD, corr, dense, tol, itnlim > 0 ? itnlim : 2000,
                                                     info, decomposition ? nullptr : j.matD);
        if (rcd != MPGPU_OK) return rcd;
        nrank = info->nrank;
    } else {
        // chdec2 + chslv2 (mpnum.f90:891-987)
        MPG_CUDA(c, cudaMemsetAsync(scal + 16, 0, sizeof(double) * 3, s));
        MPG_CUDA(c, packed_chdec_solve(nfit, j.matD, corr, scal + 16, work, s));
        double st[3];
        MPG_CUDA(c, cudaMemcpyAsync(st, scal + 16, sizeof(double) * 3, cudaMemcpyDeviceToHost, s));
        MPG_CUDA(c, cudaStreamSynchronize(s));
        info->evmax = st[0];
        info->evmin = st[1];
        nrank = (int)st[2];
    }
    info->nrank = nrank;
    if (ncon > 0 && !wyElim) {   // (the WY form returns the full correction)
        MPG_CUDA(c, cudaMemcpyAsync(corr + nfit, yv, sizeof(double) * ncon, cudaMemcpyDeviceToDevice, s));
        S.qlmlq(corr, 0);
    }
    if (!decomposition && errs) {
        // covariance Q A^-1 Q^T with the constraint rows zeroed (xloopn,
        // pede.f90:9094-9121); its diagonal gives the parameter errors
        if (ncon > 0) {
            k_zero_rows<<<S.grid(ncon, 1), kThreads, 0, s>>>(nfit, n, j.matD);
            qlssq(0);
        }
        k_get_diag<<<S.grid(n), kThreads, 0, s>>>(n, j.matD, diag);
        MPG_CUDA(c, cudaMemcpyAsync(errs, diag, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    }
    MPG_CUDA(c, cudaMemcpyAsync(corrOut, corr, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    cudaEventRecord(e1, s);
    MPG_CUDA(c, cudaStreamSynchronize(s));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    info->ms = ms;
    cudaEventDestroy(e0);
    cudaEventDestroy(e1);
    return MPGPU_OK;
}

// ---------------------------------------------------------------- MINRES
// mminrs (pede.f90:8243-8333) with the diagonal preconditioner of the
// QL-reduced matrix and MINRES (Paige & Saunders 1975) kept on the device;
// with qlp, MINRES-QLP on the same Lanczos process (mminrsqlp, the method's
// QLP steps from the first iteration, maxxnorm = nfit / sqrt(eps) as
// pede.f90:626 sets it).
int32_t solve_minres(mpgpu_ctx *c, const double *consResiduals, double rtol, int32_t itnlim,
                     double *corrOut, mpgpu_solveinfo *info, bool qlp) {
    Solver S(c);
    DevJob &j = c->j;
    cudaStream_t s = c->stream;
    const int32_t n = j.nVar, ncon = j.ncon, nfit = n - ncon;
    // released on every return
    struct Events {
        cudaEvent_t e[3] = {nullptr, nullptr, nullptr};
        ~Events() {
            for (cudaEvent_t x : e)
                if (x) cudaEventDestroy(x);
        }
    } ev;
    for (cudaEvent_t &x : ev.e) cudaEventCreate(&x);
    cudaEvent_t e0 = ev.e[0], e1 = ev.e[1], ep = ev.e[2];
    cudaEventRecord(e0, s);
    int32_t rc = S.prepare_product();
    if (rc) return rc;
    // workspace, kept by the job: vectors, partial sums, the reflections'
    // columns, the iteration's scalars
    const int64_t nv = ((int64_t)std::max(n, 1) + 1) / 2 * 2;   // vectors stay 16-byte aligned
    const int nb = (int)std::min<int64_t>(kMrBlocks, (nfit + kThreads - 1) / kThreads + (nfit < 1));
    const int nbY1 = (int)std::min<int64_t>(kMrBlocks, ((int64_t)nfit * kY1Lanes + kY1Threads - 1) / kY1Threads + (nfit < 1));
    const int nbStep = (int)std::min<int64_t>(kStepBlocks, (n + kStepRows - 1) / kStepRows);
    const int64_t nUW = (int64_t)nbStep * 2 * kWyFused;
    const int64_t scalLen = (2 * sizeof(MinresState) + 2 * sizeof(QlpState) + sizeof(MinresFlags)) / 8 + 8;
    auto padded = [&] { return S.useRows && ncon <= kWyFused ? ((int64_t)j.nG * j.br.R + 1) / 2 * 2 : nv; };
    auto grow = [&] {
        return dgrow(j, j.work, 16 * nv + padded() + 3 * kMrBlocks + kDotBlocks + 8 + nUW + 2 * kWyFused + scalLen +
                                    S.wy_len());
    };
    cudaError_t eWork = grow();
    if (eWork != cudaSuccess && S.useRows) {   // without the copy and the reflections' columns
        rc = S.from_storage();
        if (rc) return rc;
        eWork = grow();
    }
    MPG_CUDA(c, eWork);
    const bool fused = S.useRows && ncon <= kWyFused;
    const int64_t nxp = padded();
    double *at = j.work;
    auto vec = [&](int64_t l) {
        double *p = at;
        at += l;
        return p;
    };
    double *xa = vec(nxp), *rhs = vec(nv), *ba = vec(nv), *dg = vec(nv), *cu = vec(nv), *tmp = vec(nv), *yk = vec(nv);
    double *r[2] = {vec(nv), vec(nv)}, *y = vec(nv), *v = vec(nv), *w[2] = {vec(nv), vec(nv)}, *x = vec(nv);
    double *xp = vec(nv), *xc = vec(nv), *xb = vec(nv);
    double *partA = vec(kMrBlocks), *partB = vec(kMrBlocks), *partX = vec(kMrBlocks), *partD = vec(kDotBlocks + 8);
    double *partUW = vec(nUW), *coef = vec(2 * kWyFused);
    MinresState *St = reinterpret_cast<MinresState *>(at);
    QlpState *Qs = reinterpret_cast<QlpState *>(St + 2);
    MinresFlags *F = reinterpret_cast<MinresFlags *>(Qs + 2);
    at += scalLen;
    S.part = partD;
    MPG_CUDA(c, cudaMemcpyAsync(rhs, j.gvec, sizeof(double) * n, cudaMemcpyDeviceToDevice, s));
    if (S.wy_fits()) {
        rc = S.wy_build(at);
        if (rc) return rc;
    }
    std::vector<double> yc(ncon > 0 ? ncon : 1, 0.0);
    double *dsc = c->scal + 300;
    if (ncon > 0) {
        for (int k = ncon; k >= 1; --k) {
            double d = 0.0;
            for (int cc = 1; cc <= ncon - k; ++cc) d = d + j.hL[(size_t)(k - 1) * ncon + k - 1 + cc] * yc[k - 1 + cc];
            yc[k - 1] = ((consResiduals ? consResiduals[k - 1] : 0.0) - d) / j.hL[(size_t)(k - 1) * ncon + k - 1];
        }
        // rhs - A Q [0; y], then Q^T
        MPG_CUDA(c, cudaMemsetAsync(xb, 0, sizeof(double) * n, s));
        MPG_CUDA(c, cudaMemcpyAsync(xb + nfit, yc.data(), sizeof(double) * ncon, cudaMemcpyHostToDevice, s));
        S.qlmlq(xb, 0);
        S.avprd0(xb, ba);
        k_sub<<<S.grid(n), kThreads, 0, s>>>(n, rhs, ba);
        S.qlmlq(rhs, 1);
    }
    // preconditioner (pede.f90:8292-8316 by mbandw): < 0 none (M = I), 0
    // the diagonal of Q^T A Q (the band-width-1 case of qlpssq,
    // mpqldec.f90:711-950: dg -= 4 v y - 4 (v.y) v^2 per reflection), > 0
    // the variable-band Cholesky factor of its band (equdecs/equslvs)
    const int32_t mbandw = c->mbandw;
    BandPre P;
    struct BandGuard { BandPre &p; ~BandGuard() { band_free(p); } } bandGuard{P};
    if (mbandw == 0) {
        if (j.matsto == 2) k_sparse_diag<<<S.grid(n), kThreads, 0, s>>>(n, j.matD, dg);
        else k_get_diag<<<S.grid(n), kThreads, 0, s>>>(n, j.matD, dg);
        if (S.wy.m > 0)
            k_diag_eliminate<<<(n + kThreads - 1) / kThreads, kThreads, 0, s>>>(n, S.wy.m, S.wy.UWc, S.wy.Z, dg);
        else
            S.reflections(v, tmp, yk, dsc, [&] { k_diag_update<<<S.grid(n), kThreads, 0, s>>>(n, dg, v, yk, dsc); });
        k_precond<<<S.grid(nfit), kThreads, 0, s>>>(nfit, dg, cu);
    } else {
        k_fill<<<S.grid(nfit), kThreads, 0, s>>>(nfit, 1.0, cu);
        if (mbandw > 0) {
            rc = S.band_build(P, mbandw, c->lprecm, v, tmp, yk, dsc);
            if (rc) return rc;
        }
    }
    cudaEventRecord(ep, s);
    // MINRES state: x = 0, r1 = r2 = b, y = M^-1 r1, beta1 = sqrt(r1.y)
    MPG_CUDA(c, cudaMemsetAsync(x, 0, sizeof(double) * n, s));
    MPG_CUDA(c, cudaMemsetAsync(xa, 0, sizeof(double) * nxp, s));
    for (double *p : {w[0], w[1], xp}) MPG_CUDA(c, cudaMemsetAsync(p, 0, sizeof(double) * n, s));
    for (double *p : {r[0], r[1]})
        MPG_CUDA(c, cudaMemcpyAsync(p, rhs, sizeof(double) * nfit, cudaMemcpyDeviceToDevice, s));
    k_apply_precond<<<S.grid(nfit), kThreads, 0, s>>>(nfit, r[0], cu, y);
    if (mbandw > 0) MPG_CUDA(c, band_solve(P, nullptr, y, s));
    dot(r[0], y, nfit, partD, dsc, s);
    k_mr_init<<<1, 32, 0, s>>>(St, qlp ? Qs : nullptr, F, dsc, rtol, itnlim);
    const double maxxnorm = (double)nfit / sqrt(2.220446049250313e-16);
    const bool pad = fused && !j.br.uniform;
    StepParams sp{};
    sp.n = n; sp.nfit = nfit; sp.m = fused ? ncon : 0; sp.R = fused ? j.br.R : 0;
    sp.aig = pad ? j.aig : nullptr; sp.p2g = j.p2g;
    sp.F = F; sp.partB = partB; sp.y = y; sp.UWr = S.wy.UWr; sp.v = v; sp.xa = xa;
    sp.partX = partX; sp.partUW = partUW; sp.x = x; sp.xp = xp; sp.xc = xc;
    Y1Params y1{};
    y1.nfit = nfit; y1.n = n; y1.m = sp.m; y1.R = sp.R; y1.aig = j.aig; y1.p2g = j.p2g;
    y1.itemBeg = j.br.itemBeg; y1.part = j.br.part; y1.UWc = S.wy.UWc; y1.coef = coef; y1.ba = ba; y1.v = v;
    y1.xc = qlp ? xc : nullptr; y1.F = F; y1.y = y; y1.x = x; y1.partA = partA;
    BlockRowsCoef bc{sp.m, nbStep, partUW, j.qlT, S.wy.S, coef, {nullptr, F, partX, nbStep, qlp ? maxxnorm : -1.0}};
    sp.Sin = St;
    k_mr_step<kStart><<<nbStep, kThreads, 0, s>>>(sp);
    // the iterations of one batch are recorded once as a CUDA graph and
    // replayed (all scalars live on the device); direct launches if the
    // capture is refused.  An even number: the two copies of the scalars and
    // the buffer pairs have swapped back at its end.
    const int batch = 16;
    auto batchBody = [&] {
        for (int q = 0; q < batch; ++q) {
            const int a = q & 1, b = 1 - a;   // current and next scalars; older and current of r and w
            bc.test.S = St + a;
            y1.S = St + a;
            y1.r1 = r[a];
            if (fused) {
                block_rows_spmv(j.br, xa, &F->done, &bc, s);
                k_mr_y1<true><<<nbY1, kY1Threads, 0, s>>>(y1);
            } else {
                k_mr_test<<<1, 32, 0, s>>>(bc.test);
                S.qlmlq(xa, 0);
                S.avprd0(xa, ba);
                S.qlmlq(ba, 1);
                k_mr_y1<false><<<nbY1, kY1Threads, 0, s>>>(y1);
            }
            k_mr_y2<<<nb, kThreads, 0, s>>>(nfit, St + a, F, partA, nbY1, y, r[a], r[b], cu, partB);
            sp.npB = nb;
            if (mbandw > 0) {
                band_solve(P, &F->done, y, s);
                k_dot_partial<<<kDotBlocks, kThreads, 0, s>>>(nfit, r[a], y, partB);
                sp.npB = kDotBlocks;
            }
            sp.Sin = St + a; sp.Sout = St + b;
            sp.Qin = Qs + a; sp.Qout = Qs + b;
            sp.wa = qlp ? w[0] : w[a];
            sp.wb = qlp ? w[1] : w[b];
            if (qlp) k_mr_step<kQlp><<<nbStep, kThreads, 0, s>>>(sp);
            else k_mr_step<kMinres><<<nbStep, kThreads, 0, s>>>(sp);
        }
    };
    struct GraphGuard {
        cudaGraph_t g = nullptr;
        cudaGraphExec_t e = nullptr;
        ~GraphGuard() {
            if (e) cudaGraphExecDestroy(e);
            if (g) cudaGraphDestroy(g);
        }
    } gg;
    if (cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal) == cudaSuccess) {
        batchBody();
        if (cudaStreamEndCapture(s, &gg.g) != cudaSuccess || cudaGraphInstantiate(&gg.e, gg.g, 0) != cudaSuccess)
            gg.e = nullptr;
        cudaGetLastError();
    }
    MinresState hs[2];
    MinresFlags hf;
    for (int it = 0;;) {
        if (gg.e) MPG_CUDA(c, cudaGraphLaunch(gg.e, s));
        else batchBody();
        it += batch;
        MPG_CUDA(c, cudaMemcpyAsync(hs, St, sizeof(hs), cudaMemcpyDeviceToHost, s));
        MPG_CUDA(c, cudaMemcpyAsync(&hf, F, sizeof(hf), cudaMemcpyDeviceToHost, s));
        MPG_CUDA(c, cudaStreamSynchronize(s));
        if (hf.done || it > itnlim + batch) break;
    }
    const MinresState &last = hs[1].k > hs[0].k ? hs[1] : hs[0];   // the copy that the last step wrote
    info->itn = last.itn;
    info->istop = last.istop;
    if (ncon > 0) {
        MPG_CUDA(c, cudaMemcpyAsync(x + nfit, yc.data(), sizeof(double) * ncon, cudaMemcpyHostToDevice, s));
        S.qlmlq(x, 0);
    }
    MPG_CUDA(c, cudaMemcpyAsync(corrOut, x, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    cudaEventRecord(e1, s);
    MPG_CUDA(c, cudaStreamSynchronize(s));
    float ms = 0.0f;
    cudaEventElapsedTime(&ms, e0, e1);
    info->ms = ms;
    cudaEventElapsedTime(&ms, e0, ep);
    info->msFactor = ms;
    if (mbandw > 0) cudaMemcpy(&info->nrkd, P.nrkd, sizeof(int32_t), cudaMemcpyDeviceToHost);
    return MPGPU_OK;
}

int32_t avprod_host(mpgpu_ctx *c, int32_t n, const double *x, double *b) {
    Solver S(c);
    DevJob &j = c->j;
    cudaStream_t s = c->stream;
    const int32_t rcp = S.prepare_product();
    if (rcp) return rcp;
    double *xa = nullptr, *ba = nullptr;
    MPG_CUDA(c, cudaMalloc(&xa, sizeof(double) * j.nVar));
    MPG_CUDA(c, cudaMalloc(&ba, sizeof(double) * j.nVar));
    MPG_CUDA(c, cudaMemsetAsync(xa, 0, sizeof(double) * j.nVar, s));
    MPG_CUDA(c, cudaMemcpyAsync(xa, x, sizeof(double) * n, cudaMemcpyHostToDevice, s));
    S.qlmlq(xa, 0);
    S.avprd0(xa, ba);
    S.qlmlq(ba, 1);
    MPG_CUDA(c, cudaMemcpyAsync(b, ba, sizeof(double) * n, cudaMemcpyDeviceToHost, s));
    MPG_CUDA(c, cudaStreamSynchronize(s));
    cudaFree(xa);
    cudaFree(ba);
    return MPGPU_OK;
}

// the band preconditioner alone (equdecs on pede's matPreCond): band of
// Q^T A Q and its lltdec factor, returned in the variable-band layout of
// indPreCond (pede.f90:7705-7717) for the nfit rows
int32_t band_precond_factor(mpgpu_ctx *c, int32_t mbandw, int32_t lprecm, double *cOut, int32_t *nrkd) {
    Solver S(c);
    DevJob &j = c->j;
    cudaStream_t s = c->stream;
    const int32_t n = j.nVar, nfit = n - j.ncon;
    if (mbandw <= 0) return set_err(c, MPGPU_ERR_ARG, "band width must be positive");
    const int32_t rcp = S.prepare_product();
    if (rcp) return rcp;
    MPG_CUDA(c, cudaMallocAsync(&S.partOwned, sizeof(double) * (kDotBlocks + 8), s));
    S.part = S.partOwned;
    struct Bufs {
        double *v = nullptr, *tmp = nullptr, *yk = nullptr;
        BandPre P;
        ~Bufs() {
            cudaFree(v); cudaFree(tmp); cudaFree(yk);
            band_free(P);
        }
    } bb;
    double *&v = bb.v, *&tmp = bb.tmp, *&yk = bb.yk;
    MPG_CUDA(c, cudaMalloc(&v, sizeof(double) * std::max(n, 1)));
    MPG_CUDA(c, cudaMalloc(&tmp, sizeof(double) * std::max(n, 1)));
    MPG_CUDA(c, cudaMalloc(&yk, sizeof(double) * std::max(n, 1)));
    BandPre &P = bb.P;
    int32_t rc = S.band_build(P, mbandw, lprecm, v, tmp, yk, c->scal + 300);
    if (!rc) {
        const int W1 = P.w + 1;
        std::vector<double> F((size_t)std::max(nfit, 1) * W1);
        cudaMemcpyAsync(F.data(), P.F, sizeof(double) * F.size(), cudaMemcpyDeviceToHost, s);
        cudaMemcpyAsync(nrkd, P.nrkd, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
        if (cudaStreamSynchronize(s) != cudaSuccess) rc = cuda_err(c, cudaGetLastError(), "band factor");
        int64_t pos = 0;  // india(i) - i + j, 0-based running position
        for (int32_t i = 0; !rc && i < nfit; ++i)
            for (int32_t t = std::max(0, P.w - i); t <= P.w; ++t) cOut[pos++] = F[(size_t)i * W1 + t];
    }
    return rc;
}
