// mpgpu_bspmv.cu -- y = A x for the mpbits-sparse matrix (avprd0,
// pede.f90:5069-5358) from a symmetric block-row copy.
//
// Bound: FP64.  Every stored off-diagonal element takes two fused
// multiply-adds and GB300 issues two FP64 lanes per SM and clock, so 9.0M
// stored elements (5,000 barrel modules, 400,000 tracks) take 28.6 us at 2.07
// GHz; the copy holds each block with its transpose (144 MB there), 21 us of
// HBM traffic underneath.  The first form read the storage once and summed
// transposed products through a buffer (46 us and 51 us passes): the second
// pass and its shuffle trees were the larger half.
//
// Layout: a row group's blocks (its own, its diagonal block, the transposed
// incoming ones, by ascending column group) are cut into steps of nslot = 32 /
// R blocks.  Lane slot * R + ii owns row ii of the step's block `slot`, so a
// step is R fused multiply-adds per lane with 30 of 32 lanes busy for R = 6,
// and no sum crosses lanes inside an item; the step's values are stored in
// lane order (two columns per lane for even R: 16-byte loads).  Items of at
// most itemSteps steps of one row group go to one warp each; their sums are
// added in item order.  No atomics, fixed order: the product is reproducible.
// 9.0M
// stored elements: 44 us (FP64 pipe 83 % busy while the SMs are active),
// 6.9M: 35 us (first form 101 and 84 us).
#include <algorithm>
#include <vector>

#include "mpgpu_bspmv.h"
#include "mpgpu_records.cuh"

namespace {

constexpr int kBrMax = 8;        // parameters per group
constexpr int kBrWarps = 8;      // warps per CTA of the product
constexpr int kBrUnroll = 4;     // steps whose loads are in flight together

// per row group: its stored off-diagonal blocks in list order (ownBlk), its
// diagonal block (diagBlk, -1: none stored); per block its column group as a
// sort key (nG + 1 for blocks that are not transposed) and itself as value
__global__ void k_br_own(int32_t nG, int64_t nmat, const int64_t *rowBlk0, const int32_t *blkJ, const int64_t *blkOff,
                         int32_t *ownBlk, int32_t *own, int32_t *diagBlk, int32_t *brow, uint64_t *key,
                         uint32_t *val) {
    const int ln = threadIdx.x & 31;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t I = 1 + w; I <= nG; I += nw) {
        const int64_t b0 = rowBlk0[I - 1], b1 = rowBlk0[I];
        int n = 0;
        int32_t diag = -1;
        for (int64_t q = b0; q < b1; q += 32) {
            const int64_t b = q + ln;
            const bool stored = b < b1 && blkOff[b] < nmat;   // beyond: the discard area of left-out pairs
            const int32_t J = b < b1 ? blkJ[b] : 0;
            const bool off = stored && J != I;
            const unsigned m = __ballot_sync(kFull, off);
            const unsigned d = __ballot_sync(kFull, stored && J == I);
            if (off) ownBlk[b0 + n + __popc(m & ((1u << ln) - 1u))] = (int32_t)b;
            n += __popc(m);
            if (d) diag = (int32_t)(q + __ffs(d) - 1);
            if (b < b1) {
                brow[b] = (int32_t)I;
                key[b] = off ? (uint64_t)J : (uint64_t)(nG + 1);
                val[b] = (uint32_t)b;
            }
        }
        if (ln == 0) {
            own[I - 1] = n;
            diagBlk[I - 1] = diag;
        }
    }
}

// range of every column group in the sorted keys
__global__ void k_br_incoming(const uint64_t *key, int64_t n, int32_t nG, int64_t *beg, int64_t *end) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n || key[i] > (uint64_t)nG) return;
    if (i == 0 || key[i - 1] != key[i]) beg[key[i] - 1] = i;
    if (i == n - 1 || key[i + 1] != key[i]) end[key[i] - 1] = i + 1;
}

__global__ void k_br_steps(int32_t nG, int nslot, const int32_t *own, const int64_t *beg, const int64_t *end,
                           int64_t *steps) {
    const int64_t I = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (I > nG) return;
    steps[I] = I < nG ? (own[I] + 1 + (end[I] - beg[I]) + nslot - 1) / nslot : 0;
}

__global__ void k_br_nitems(int32_t nG, int itemSteps, const int64_t *stepBeg, int64_t *items) {
    const int64_t I = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (I > nG) return;
    items[I] = I < nG ? (stepBeg[I + 1] - stepBeg[I] + itemSteps - 1) / itemSteps : 0;
}

__global__ void k_br_items(int32_t nG, int itemSteps, const int64_t *stepBeg, const int64_t *itemBeg, int32_t *s0,
                           int32_t *s1) {
    const int64_t I = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (I >= nG) return;
    const int64_t a = stepBeg[I], e = stepBeg[I + 1];
    for (int64_t k = itemBeg[I]; k < itemBeg[I + 1]; ++k) {
        const int64_t q = a + (k - itemBeg[I]) * itemSteps;
        s0[k] = (int32_t)q;
        s1[k] = (int32_t)min(e, q + itemSteps);
    }
}

struct BrFill {
    int32_t nG;
    int64_t nsteps;
    const int64_t *rowBlk0, *stepBeg, *beg, *end, *blkOff;
    const int32_t *ownBlk, *own, *diagBlk, *brow, *blkJ, *blkLd, *aig;
    const uint32_t *sorted;
    const double *matD;
};

// one warp per step: the column groups and values of its nslot blocks
template <int R>
__global__ void k_br_fill(BrFill P, int32_t *col, double *val) {
    constexpr int NS = 32 / R, L = NS * R;
    const int ln = threadIdx.x & 31, slot = ln / R, ii = ln - slot * R;
    const int64_t w = ((int64_t)blockIdx.x * blockDim.x + threadIdx.x) >> 5;
    const int64_t nw = ((int64_t)gridDim.x * blockDim.x) >> 5;
    for (int64_t t = w; t < P.nsteps; t += nw) {
        if (ln >= L) continue;
        int64_t lo = 0, hi = P.nG - 1;
        while (lo < hi) {
            const int64_t mid = (lo + hi + 1) >> 1;
            if (P.stepBeg[mid] <= t) lo = mid;
            else hi = mid - 1;
        }
        const int64_t I = lo;   // 0-based row group
        const int64_t e = (t - P.stepBeg[I]) * NS + slot;
        const int64_t own = P.own[I], inc = P.end[I] - P.beg[I];
        const int32_t ia = P.aig[I] - 1, np = P.aig[I + 1] - 1 - ia;
        int64_t J = I, b = -1;
        int kind = 0;   // 0 padding, 1 own, 2 diagonal, 3 incoming (transposed)
        if (e < own) {
            kind = 1;
            b = P.ownBlk[P.rowBlk0[I] + e];
            J = P.blkJ[b] - 1;
        } else if (e == own) {
            kind = 2;
            b = P.diagBlk[I];
        } else if (e <= own + inc) {
            kind = 3;
            b = P.sorted[P.beg[I] + e - own - 1];
            J = P.brow[b] - 1;
        }
        const int32_t nj = P.aig[J + 1] - P.aig[J];
        const int64_t off = b >= 0 ? P.blkOff[b] : 0, ld = b >= 0 ? P.blkLd[b] : 0;
        if (ii == 0) col[t * NS + slot] = (int32_t)J;
#pragma unroll
        for (int jj = 0; jj < R; ++jj) {
            double v = 0.0;
            if (ii < np && jj < nj) {
                if (kind == 1) v = P.matD[off + ii * ld + jj];
                else if (kind == 3) v = P.matD[off + jj * ld + ii];
                else if (kind == 2) {
                    if (ii == jj) v = P.matD[ia + ii];
                    else if (b >= 0) v = P.matD[off + max(ii, jj) * ld + min(ii, jj)];
                }
            }
            const int64_t at = R % 2 == 0 ? ((t * (R / 2) + jj / 2) * L + ln) * 2 + jj % 2 : (t * R + jj) * L + ln;
            val[at] = v;
        }
    }
}

// coefficients of the constraint reflections from the partial dots: with s =
// U^T x, t = W^T x: a = T^T s, c = T t - S s
__device__ void br_coef(const BlockRowsCoef &k) {
    extern __shared__ double sc[];   // 2 m sums, then the partial sums
    const int C = 2 * k.m, tid = threadIdx.x;
    mr_test(k.test);
    if (C == 0) return;
    const int nsub = blockDim.x / C, sub = tid / C, cc = tid - sub * C;
    double *red = sc + C;
    if (sub < nsub) {
        double v0 = 0.0, v1 = 0.0, v2 = 0.0, v3 = 0.0;
        int b = sub;
        for (; b + 3 * nsub < k.nblk; b += 4 * nsub) {
            v0 += k.partUW[(int64_t)b * C + cc];
            v1 += k.partUW[(int64_t)(b + nsub) * C + cc];
            v2 += k.partUW[(int64_t)(b + 2 * nsub) * C + cc];
            v3 += k.partUW[(int64_t)(b + 3 * nsub) * C + cc];
        }
        for (; b < k.nblk; b += nsub) v0 += k.partUW[(int64_t)b * C + cc];
        red[sub * C + cc] = (v0 + v1) + (v2 + v3);
    }
    __syncthreads();
    if (tid < C) {
        double v = 0.0;
        for (int q = 0; q < nsub; ++q) v += red[q * C + tid];
        sc[tid] = v;
    }
    __syncthreads();
    if (tid < k.m) {
        double v = 0.0;
        for (int q = tid; q < k.m; ++q) v = fma(k.T[tid * k.m + q], sc[k.m + q], v);
        for (int q = 0; q < k.m; ++q) v = fma(-k.S[tid * k.m + q], sc[q], v);
        k.coef[tid] = v;
    } else if (tid < C) {
        const int r = tid - k.m;
        double v = 0.0;
        for (int q = 0; q <= r; ++q) v = fma(k.T[q * k.m + r], sc[q], v);
        k.coef[tid] = v;
    }
}

// a lane's R values of one step (column pairs for even R) and the R values of x
template <int R>
__device__ __forceinline__ void br_load(const double *p, double (&v)[R]) {
    constexpr int L = 32 / R * R;
    if constexpr (R % 2 == 0) {
#pragma unroll
        for (int q = 0; q < R / 2; ++q)
            asm("ld.global.nc.L1::no_allocate.v2.f64 {%0, %1}, [%2];"
                : "=d"(v[2 * q]), "=d"(v[2 * q + 1])
                : "l"(p + q * 2 * L));
    } else {
#pragma unroll
        for (int q = 0; q < R; ++q)
            asm("ld.global.nc.L1::no_allocate.f64 %0, [%1];" : "=d"(v[q]) : "l"(p + q * L));
    }
}
template <int R>
__device__ __forceinline__ void br_load_x(const double *p, double (&x)[R]) {
    if constexpr (R % 2 == 0) {
#pragma unroll
        for (int q = 0; q < R / 2; ++q) {
            const double2 y = __ldg(reinterpret_cast<const double2 *>(p) + q);
            x[2 * q] = y.x;
            x[2 * q + 1] = y.y;
        }
    } else {
#pragma unroll
        for (int q = 0; q < R; ++q) x[q] = __ldg(p + q);
    }
}

template <int R, bool COEF>
__global__ void __launch_bounds__(32 * kBrWarps) k_br_spmv(int64_t nitem, const int32_t *s0, const int32_t *s1,
                                                           const int32_t *col, const double *val, const double *xp,
                                                           double *part, const int32_t *done, BlockRowsCoef coef) {
    constexpr int NS = 32 / R, L = NS * R;
    if (done && *done) return;
    if (COEF && blockIdx.x == 0) {
        br_coef(coef);
        return;
    }
    const int ln = threadIdx.x & 31, slot = ln / R;
    const int64_t it = (int64_t)(blockIdx.x - (COEF ? 1 : 0)) * kBrWarps + (threadIdx.x >> 5);
    if (it >= nitem) return;
    const int a = s0[it], e = s1[it];
    double acc0 = 0.0, acc1 = 0.0;
    if (ln < L) {
        const int32_t *cp = col + (int64_t)a * NS + slot;
        const double *vp = val + (int64_t)a * R * L + (R % 2 == 0 ? 2 * ln : ln);
        // kBrUnroll steps' loads in flight together: columns, then values and x
        auto steps = [&](auto cnt) {
            constexpr int U = decltype(cnt)::value;
            int32_t c[U];
            double v[U][R], x[U][R];
#pragma unroll
            for (int u = 0; u < U; ++u) c[u] = __ldg(cp + u * NS);
#pragma unroll
            for (int u = 0; u < U; ++u) br_load<R>(vp + u * R * L, v[u]);
#pragma unroll
            for (int u = 0; u < U; ++u) br_load_x<R>(xp + (int64_t)c[u] * R, x[u]);
#pragma unroll
            for (int u = 0; u < U; ++u)
#pragma unroll
                for (int q = 0; q < R; ++q) {
                    if (q % 2 == 0) acc0 = fma(v[u][q], x[u][q], acc0);
                    else acc1 = fma(v[u][q], x[u][q], acc1);
                }
            cp += U * NS;
            vp += U * R * L;
        };
        int t = a;
        for (; t + kBrUnroll <= e; t += kBrUnroll) steps(std::integral_constant<int, kBrUnroll>());
        for (; t < e; ++t) steps(std::integral_constant<int, 1>());
    }
    double v = acc0 + acc1;
    if constexpr ((R & (R - 1)) == 0) {
#pragma unroll
        for (int o = R; o < 32; o *= 2) v += __shfl_xor_sync(kFull, v, o);
    } else {
        const double mine = v;
#pragma unroll
        for (int q = 1; q < NS; ++q) v += __shfl_sync(kFull, mine, (ln + q * R) & 31);   // used by lanes < R
    }
    if (ln < R) part[it * R + ln] = v;
}

__global__ void k_br_pad(int32_t n, int R, const int32_t *aig, const int32_t *p2g, const double *x, double *xp) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t g = p2g[i] - 1;
    xp[(int64_t)g * R + i - (aig[g] - 1)] = x[i];
}

__global__ void k_br_sum(int32_t n, int R, const int32_t *aig, const int32_t *p2g, const int64_t *itemBeg,
                         const double *part, double *y) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    const int32_t g = p2g[i] - 1;
    const int64_t ii = i - (aig[g] - 1);
    double v = 0.0;
    for (int64_t k = itemBeg[g]; k < itemBeg[g + 1]; ++k) v += part[k * R + ii];
    y[i] = v;
}

template <class F>
void by_group_size(int R, F &&f) {
    switch (R) {
    case 1: f(std::integral_constant<int, 1>()); break;
    case 2: f(std::integral_constant<int, 2>()); break;
    case 3: f(std::integral_constant<int, 3>()); break;
    case 4: f(std::integral_constant<int, 4>()); break;
    case 5: f(std::integral_constant<int, 5>()); break;
    case 6: f(std::integral_constant<int, 6>()); break;
    case 7: f(std::integral_constant<int, 7>()); break;
    default: f(std::integral_constant<int, 8>()); break;
    }
}

int max_group(const std::vector<int32_t> &aig, int *minOut) {
    int mx = 0, mn = 1 << 30;
    for (size_t g = 1; g < aig.size(); ++g) {
        mx = std::max(mx, aig[g] - aig[g - 1]);
        mn = std::min(mn, aig[g] - aig[g - 1]);
    }
    if (minOut) *minOut = mn;
    return mx;
}

}  // namespace

// The copy is taken when its padding costs less than the second pass it
// saves: groups of one size need none; mixed sizes up to 1.6 times the
// stored elements.
bool block_rows_fit(const mpgpu_ctx *c) {
    const DevJob &j = c->j;
    if (j.matsto != 2 || j.nG <= 0) return false;
    int mn = 0;
    const int R = max_group(j.hAig, &mn);
    const int64_t nblk = (int64_t)j.hBlkJ.size();
    if (R < 1 || R > kBrMax || nblk >= ((int64_t)1 << 31) - 2) return false;
    return mn == R || (double)(nblk + j.nG) * R * R <= 1.6 * (double)j.nmat;
}

int32_t block_rows_build(mpgpu_ctx *c) {
    DevJob &j = c->j;
    BlockRows &b = j.br;
    cudaStream_t s = c->stream;
    b.R = 0;
    int nsm = 0;
    MPG_CUDA(c, cudaDeviceGetAttribute(&nsm, cudaDevAttrMultiProcessorCount, c->device));
    int mn = 0;
    const int R = max_group(j.hAig, &mn), NS = 32 / R, L = NS * R;
    const int32_t nG = j.nG;
    const int64_t nblk = (int64_t)j.hBlkJ.size(), nsort = std::max<int64_t>(nblk, 1);
    b.nG = nG;
    b.nVar = j.nVar;
    b.nslot = NS;
    b.uniform = mn == R;
    // scratch of the set-up, one allocation
    struct Scratch {
        char *p = nullptr;
        cudaStream_t s;
        ~Scratch() { if (p) cudaFreeAsync(p, s); }
    } W{nullptr, s};
    const int64_t ntile = (nsort + kRsTile - 1) / kRsTile;
    const int64_t scanLen = scan_tmp_len(std::max<int64_t>(256 * ntile + 1, nG + 1));
    int64_t at = 0;
    auto take = [&](int64_t bytes) {
        const int64_t o = at;
        at += (bytes + 255) / 256 * 256;
        return o;
    };
    const int64_t oK0 = take(8 * nsort), oK1 = take(8 * nsort), oV0 = take(4 * nsort), oV1 = take(4 * nsort),
                  oH = take(8 * (256 * ntile + 1)), oT = take(8 * std::max<int64_t>(scanLen, 1)), oOwn = take(4 * nsort),
                  oBrow = take(4 * nsort), oN = take(4 * (int64_t)nG), oD = take(4 * (int64_t)nG),
                  oB = take(8 * (int64_t)nG), oE = take(8 * (int64_t)nG), oC = take(8 * ((int64_t)nG + 1));
    MPG_CUDA(c, cudaMallocAsync((void **)&W.p, (size_t)at, s));
    uint64_t *k0 = (uint64_t *)(W.p + oK0), *k1 = (uint64_t *)(W.p + oK1);
    uint32_t *v0 = (uint32_t *)(W.p + oV0), *v1 = (uint32_t *)(W.p + oV1);
    int32_t *ownBlk = (int32_t *)(W.p + oOwn), *brow = (int32_t *)(W.p + oBrow), *own = (int32_t *)(W.p + oN),
            *diag = (int32_t *)(W.p + oD);
    int64_t *beg = (int64_t *)(W.p + oB), *end = (int64_t *)(W.p + oE), *cnt = (int64_t *)(W.p + oC),
            *tmp = (int64_t *)(W.p + oT);
    MPG_CUDA(c, dgrow(j, b.stepBeg, (int64_t)nG + 1));
    MPG_CUDA(c, dgrow(j, b.itemBeg, (int64_t)nG + 1));
    k_br_own<<<blocks_for(32 * (int64_t)nG), 256, 0, s>>>(nG, j.nmat, j.rowBlk0, j.blkJ, j.blkOff, ownBlk, own, diag,
                                                          brow, k0, v0);
    SortBufs sb{k0, k1, v0, v1, (int64_t *)(W.p + oH), tmp};
    MPG_CUDA(c, radix_sort(sb, nblk, bits_for((uint64_t)nG + 1), s));
    MPG_CUDA(c, cudaMemsetAsync(beg, 0, sizeof(int64_t) * nG, s));
    MPG_CUDA(c, cudaMemsetAsync(end, 0, sizeof(int64_t) * nG, s));
    if (nblk > 0) k_br_incoming<<<blocks_for(nblk), 256, 0, s>>>(sb.k0, nblk, nG, beg, end);
    k_br_steps<<<blocks_for(nG + 1), 256, 0, s>>>(nG, NS, own, beg, end, cnt);
    MPG_CUDA(c, scan_ex(cnt, b.stepBeg, nG + 1, tmp, s));
    int64_t nsteps = 0;
    MPG_CUDA(c, cudaMemcpyAsync(&nsteps, b.stepBeg + nG, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    MPG_CUDA(c, cudaStreamSynchronize(s));
    if (nsteps >= (int64_t)1 << 31) return set_err(c, MPGPU_ERR_LIMIT, "sparse product: too many blocks");
    // steps per item: one item for every warp that fits on the device, so
    // that the sums across lanes (4 of them for R = 6) stay a small part;
    // between 4 and 16 steps, whole rounds of loads
    const int itemSteps =
        (int)std::min<int64_t>(16, std::max<int64_t>(1, (nsteps / ((int64_t)nsm * 64) + 2) / kBrUnroll) * kBrUnroll);
    k_br_nitems<<<blocks_for(nG + 1), 256, 0, s>>>(nG, itemSteps, b.stepBeg, cnt);
    MPG_CUDA(c, scan_ex(cnt, b.itemBeg, nG + 1, tmp, s));
    int64_t nitem = 0;
    MPG_CUDA(c, cudaMemcpyAsync(&nitem, b.itemBeg + nG, sizeof(int64_t), cudaMemcpyDeviceToHost, s));
    MPG_CUDA(c, cudaStreamSynchronize(s));
    MPG_CUDA(c, dgrow(j, b.val, nsteps * R * L));
    MPG_CUDA(c, dgrow(j, b.col, nsteps * NS));
    MPG_CUDA(c, dgrow(j, b.itemS0, nitem));
    MPG_CUDA(c, dgrow(j, b.itemS1, nitem));
    MPG_CUDA(c, dgrow(j, b.part, nitem * R));
    MPG_CUDA(c, dgrow(j, b.xp, (int64_t)nG * R));
    MPG_CUDA(c, cudaMemsetAsync(b.xp, 0, sizeof(double) * (size_t)nG * R, s));
    k_br_items<<<blocks_for(nG), 256, 0, s>>>(nG, itemSteps, b.stepBeg, b.itemBeg, b.itemS0, b.itemS1);
    const BrFill F{nG, nsteps, j.rowBlk0, b.stepBeg, beg, end, j.blkOff, ownBlk, own, diag, brow, j.blkJ, j.blkLd,
                   j.aig, sb.v0, j.matD};
    const unsigned fb = (unsigned)std::min<int64_t>((nsteps + 7) / 8, (int64_t)nsm * 64);
    by_group_size(R, [&](auto r) { k_br_fill<decltype(r)::value><<<fb, 256, 0, s>>>(F, b.col, b.val); });
    MPG_CUDA(c, cudaGetLastError());
    b.R = R;
    b.nsteps = nsteps;
    b.nitem = nitem;
    return MPGPU_OK;
}

int64_t block_rows_bytes(const BlockRows &b) {
    if (b.R <= 0) return 0;
    const int64_t L = (int64_t)b.nslot * b.R;
    return 8 * b.nsteps * b.R * L + 4 * b.nsteps * b.nslot + (8 * (int64_t)b.R + 8) * b.nitem +
           (16 + 8 * (int64_t)b.R) * b.nG;
}

void block_rows_free(DevJob &j) {
    BlockRows &b = j.br;
    for (void *p : {(void *)b.val, (void *)b.col, (void *)b.stepBeg, (void *)b.itemBeg, (void *)b.itemS0,
                    (void *)b.itemS1, (void *)b.part, (void *)b.xp})
        if (p) cudaFree(p);
    b = BlockRows();
}

cudaError_t block_rows_spmv(const BlockRows &b, const double *xp, const int32_t *done, const BlockRowsCoef *coef,
                            cudaStream_t s) {
    const unsigned g = (unsigned)((b.nitem + kBrWarps - 1) / kBrWarps);
    by_group_size(b.R, [&](auto r) {
        constexpr int R = decltype(r)::value;
        if (coef) {
            const int C = 2 * coef->m;
            const size_t sm = sizeof(double) * (C > 0 ? C + 32 * kBrWarps : 1);
            k_br_spmv<R, true><<<g + 1, 32 * kBrWarps, sm, s>>>(b.nitem, b.itemS0, b.itemS1, b.col, b.val, xp, b.part,
                                                                done, *coef);
        } else {
            k_br_spmv<R, false><<<g, 32 * kBrWarps, 0, s>>>(b.nitem, b.itemS0, b.itemS1, b.col, b.val, xp, b.part,
                                                            done, BlockRowsCoef{});
        }
    });
    return cudaGetLastError();
}

cudaError_t block_rows_product(const BlockRows &b, const int32_t *aig, const int32_t *p2g, const double *x, double *y,
                               cudaStream_t s) {
    const double *xp = x;
    const bool direct = b.uniform && (reinterpret_cast<uintptr_t>(x) & 15) == 0;
    if (!direct) {
        k_br_pad<<<blocks_for(b.nVar), 256, 0, s>>>(b.nVar, b.R, aig, p2g, x, b.xp);
        xp = b.xp;
    }
    const cudaError_t e = block_rows_spmv(b, xp, nullptr, nullptr, s);
    if (e != cudaSuccess) return e;
    k_br_sum<<<blocks_for(b.nVar), 256, 0, s>>>(b.nVar, b.R, aig, p2g, b.itemBeg, b.part, y);
    return cudaGetLastError();
}
