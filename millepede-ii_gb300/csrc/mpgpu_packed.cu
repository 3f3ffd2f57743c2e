// mpgpu_packed.cu -- pede's own inversion (sqminl) and decomposition (chdec2,
// chslv2) of the packed symmetric matrix, in blocks of kPb pivots.
//
// Both sweep the matrix once per pivot with a rank-1 update, in the
// reference's order.  One launch pair per pivot was bound by launches and by
// reading and writing the whole matrix for one multiply-add per element
// (1,500 rows: 27 us per pivot, 9 MB twice).  Here a panel kernel forms the
// rows of kPb pivots in turn, each brought up to date with the pivots of its
// block before it, and one update kernel then applies the block's pivots to
// every element in their order: the same operations on every element in the
// same order as pivot by pivot, with kPb multiply-adds per element read and
// written.  The update is FP64-bound (n^3 / 2 multiply-adds for sqminl, n^3 /
// 6 for chdec2 at 2 per SM and clock), the panels are bound by the latency of
// a chain of pivots.  Measured: sqminl of 1,500 rows 10.0 ms (per block 143 us
// panel, 71 us update) from 40.5 ms; chdec2 and chslv2 of 2,000 rows 5.3 ms
// (per block 22 + 11 us panel, 46 us update) from 64 ms.
#include <cooperative_groups.h>

#include <algorithm>

#include "mpgpu_fp64.cuh"
#include "mpgpu_packed.h"

namespace cg = cooperative_groups;

namespace {

constexpr int kPb = 32;        // pivots per block
constexpr int kTile = 64;      // update tiles

__device__ __forceinline__ int64_t prow(int64_t r) { return r * (r + 1) / 2; }   // offset of row r

// tile (bi, bj <= bi) of the lower triangle
__device__ __forceinline__ void tri_tile(int64_t t, int &bi, int &bj) {
    int i = (int)((sqrt(8.0 * (double)t + 1.0) - 1.0) * 0.5);
    while ((int64_t)i * (i + 1) / 2 > t) i--;
    while ((int64_t)(i + 1) * (i + 2) / 2 <= t) i++;
    bi = i;
    bj = (int)(t - (int64_t)i * (i + 1) / 2);
}

// ------------------------------------------------------------ sqminl
// Panel state: the pivots of the block and how many there are.
struct SqState {
    int32_t k[kPb];
    double vkk[kPb];
    int32_t count, stop;
};

// Rows of a CTA: warps of 32 rows dealt to the CTAs in turn.
struct SqParams {
    int32_t n, tmax;
    const double *V, *diag;
    double *b, *d;             // right-hand side, current diagonal
    int32_t *used;
    int8_t *step;              // pivot step of a row in this block (-1: none)
    double *S, *C;             // [kPb][n] scaled and unscaled pivot columns
    SqState *st;
    int32_t *deficit;
};

constexpr int kSqThreads = 256;

// One cluster takes the pivots of a block.  Per pivot: the candidates of the
// CTAs (largest |d_j| above 1e-10 of the original diagonal, lowest index on
// ties: the choice of the reference's scan) are exchanged through distributed
// shared memory with one cluster barrier; every thread then brings its rows of
// the pivot column up to date with the block's earlier pivots, scales them and
// updates its diagonal elements, so that the next choice needs no pass over
// the matrix.
__global__ void __launch_bounds__(kSqThreads) k_sqminl_panel(SqParams p) {
    cg::cluster_group cl = cg::this_cluster();
    struct Msg {
        unsigned long long bits;
        double d, b;
        int k;
    };
    __shared__ Msg msg[2];
    __shared__ unsigned long long wbits[kSqThreads / 32];
    __shared__ int wk[kSqThreads / 32];
    __shared__ double Sk[kPb], Ck[kPb], sv[2];
    __shared__ int spiv;
    const int tid = threadIdx.x, ln = tid & 31, wib = tid >> 5;
    const int nc = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int n = p.n, rowStep = nc * kSqThreads;
    const int row0 = (wib * nc + rank) * 32 + ln;
    if (p.st->stop) {   // uniform: set by an earlier launch
        if (rank == 0 && tid == 0) p.st->count = 0;   // nothing for this block's update
        return;
    }
    for (int j = row0; j < n; j += rowStep) p.step[j] = -1;
    int t = 0;
    for (; t < p.tmax; ++t) {
        unsigned long long best = 0;
        int bk = -1;
        for (int j = row0; j < n; j += rowStep) {
            if (p.used[j]) continue;
            const double a = fabs(p.d[j]);
            const unsigned long long ab = (unsigned long long)__double_as_longlong(a);
            if (a > 1.0E-10 * p.diag[j] && (bk < 0 || ab > best)) { best = ab; bk = j; }
        }
        auto take = [&](unsigned long long ob, int ok) {
            if (ok >= 0 && (bk < 0 || ob > best || (ob == best && ok < bk))) { best = ob; bk = ok; }
        };
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const unsigned long long ob = __shfl_xor_sync(0xffffffffu, best, o);
            const int ok = __shfl_xor_sync(0xffffffffu, bk, o);
            take(ob, ok);
        }
        if (ln == 0) { wbits[wib] = best; wk[wib] = bk; }
        __syncthreads();
        if (tid == 0) {
#pragma unroll
            for (int w = 1; w < kSqThreads / 32; ++w) take(wbits[w], wk[w]);
            Msg &m = msg[t & 1];
            m.bits = best;
            m.k = bk;
            m.d = bk >= 0 ? p.d[bk] : 0.0;
            m.b = bk >= 0 ? p.b[bk] : 0.0;
        }
        cl.sync();
        if (wib == 0) {
            Msg m{0, 0.0, 0.0, -1};
            if (ln < nc) m = *cl.map_shared_rank(&msg[t & 1], ln);
            best = m.bits;
            bk = m.k;
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) {
                const unsigned long long ob = __shfl_xor_sync(0xffffffffu, best, o);
                const int ok = __shfl_xor_sync(0xffffffffu, bk, o);
                take(ob, ok);
            }
            const unsigned own = __ballot_sync(0xffffffffu, bk >= 0 && m.k == bk);
            const int src = own ? __ffs(own) - 1 : 0;
            const double dk = __shfl_sync(0xffffffffu, m.d, src), bb = __shfl_sync(0xffffffffu, m.b, src);
            if (ln == 0) {
                const double vkk = bk >= 0 ? 1.0 / dk : 0.0;
                spiv = bk;
                sv[0] = vkk;
                sv[1] = bb * vkk;
                if (rank == 0) {
                    p.st->k[t] = bk;
                    p.st->vkk[t] = vkk;
                }
            }
            // the earlier pivots' columns at row k (other CTAs' writes: past L1)
            if (bk >= 0 && ln < t) {
                Sk[ln] = __ldcg(p.S + (int64_t)ln * n + bk);
                Ck[ln] = __ldcg(p.C + (int64_t)ln * n + bk);
            }
        }
        __syncthreads();
        const int k = spiv;
        if (k < 0) break;
        const double vkk = sv[0], bnew = sv[1];
        for (int j = row0; j < n; j += rowStep) {
            const int64_t at = (int64_t)t * n + j;
            if (j == k) {
                p.S[at] = 0.0;
                p.C[at] = 0.0;
                p.step[j] = (int8_t)t;
                p.used[j] = 1;
                p.b[j] = bnew;
                continue;
            }
            const int ps = p.step[j];
            double w = ps < 0 ? p.V[j > k ? prow(j) + k : prow(k) + j] : Sk[ps];
            if (j > k) {
#pragma unroll 4
                for (int q = ps + 1; q < t; ++q) w = fma(-Sk[q], p.C[(int64_t)q * n + j], w);
            } else {
#pragma unroll 4
                for (int q = ps + 1; q < t; ++q) w = fma(-p.S[(int64_t)q * n + j], Ck[q], w);
            }
            const double sc = w * vkk;
            p.S[at] = sc;
            p.C[at] = w;
            p.b[j] = fma(-bnew, w, p.b[j]);
            if (!p.used[j]) p.d[j] = fma(-sc, w, p.d[j]);
        }
        // (the next candidates read this thread's own rows only)
    }
    if (rank == 0 && tid == 0) {
        p.st->count = t;
        if (t < p.tmax) {
            p.st->stop = 1;
            *p.deficit = -1;
        }
    }
    cl.sync();   // no CTA leaves while another may read its messages
}

// The same where every thread has one row (n up to threads x CTAs of the
// cluster): the row's state stays in registers, its columns of the block in
// shared memory, where the other CTAs read the pivot row's.  The candidates are
// pushed to every CTA before the one cluster barrier of a pivot, after which
// each warp picks the pivot for itself.  (One barrier per launch besides, so
// that no CTA is pushed to before it has started.)  Bound: the chain of a pivot (exchange,
// barrier, the pivot column's element from L2, up to 31 dependent multiply-
// adds); 9.3 us per pivot with the state in global memory, now 4.5 (1,500
// rows).
struct SqMsg {
    unsigned long long bits;   // |d|
    double d, b;
    long long k;
};

__device__ __forceinline__ SqMsg sq_better(const SqMsg &x, int o) {
    SqMsg y;
    y.bits = __shfl_xor_sync(0xffffffffu, x.bits, o);
    y.d = __shfl_xor_sync(0xffffffffu, x.d, o);
    y.b = __shfl_xor_sync(0xffffffffu, x.b, o);
    y.k = __shfl_xor_sync(0xffffffffu, x.k, o);
    const bool take = y.k >= 0 && (x.k < 0 || y.bits > x.bits || (y.bits == x.bits && y.k < x.k));
    return take ? y : x;
}

template <int THREADS>
__global__ void __launch_bounds__(THREADS) k_sqminl_panel_sm(SqParams p) {
    extern __shared__ __align__(16) double hist[];   // S, then C: [kPb][THREADS]
    double *hS = hist, *hC = hist + kPb * THREADS;
    constexpr int kW = THREADS / 32;
    __shared__ SqMsg wmsg[kW], inbox[2][16];
    cg::cluster_group cl = cg::this_cluster();
    const int tid = threadIdx.x, ln = tid & 31, wib = tid >> 5;
    const int nc = (int)cl.num_blocks(), rank = (int)cl.block_rank();
    const int n = p.n, j = (wib * nc + rank) * 32 + ln;
    if (p.st->stop) {   // uniform: set by an earlier launch
        if (rank == 0 && tid == 0) p.st->count = 0;
        return;
    }
    const bool in = j < n;
    bool used = !in || p.used[j] != 0;
    double dj = in ? p.d[j] : 0.0, bj = in ? p.b[j] : 0.0;
    const double lim = in ? 1.0E-10 * p.diag[j] : 0.0;
    int ps = -1;
    int t = 0;
    cl.sync();   // every CTA runs: the first candidates are pushed before any other barrier
    for (; t < p.tmax; ++t) {
        SqMsg m{(unsigned long long)__double_as_longlong(fabs(dj)), dj, bj, j};
        if (used || !(fabs(dj) > lim)) m.k = -1;
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) m = sq_better(m, o);
        if (ln == 0) wmsg[wib] = m;
        __syncthreads();
        if (wib == 0) {
            m = wmsg[ln % kW];
#pragma unroll
            for (int o = kW / 2; o > 0; o >>= 1) m = sq_better(m, o);
            if (ln < nc) *cl.map_shared_rank(&inbox[t & 1][rank], ln) = m;
        }
        cl.sync();
        m = inbox[t & 1][ln % nc];   // nc: a power of two
        for (int o = nc / 2; o > 0; o >>= 1) m = sq_better(m, o);
        const int k = (int)m.k;
        if (k < 0) break;
        // the pivot row's earlier columns, and this row's element of column k
        double sk = 0.0, ck = 0.0;
        const int wk = k >> 5, tk = (wk / nc) * 32 + (k & 31);
        if (ln < t) {
            sk = *cl.map_shared_rank(hS + ln * THREADS + tk, wk % nc);
            ck = *cl.map_shared_rank(hC + ln * THREADS + tk, wk % nc);
        }
        double w = 0.0;
        if (in && ps < 0 && j != k) w = p.V[j > k ? prow(j) + k : prow(k) + j];
        const double vkk = 1.0 / m.d, bnew = m.b * vkk;
        if (rank == 0 && tid == 0) {
            p.st->k[t] = k;
            p.st->vkk[t] = vkk;
        }
        const double s0 = __shfl_sync(0xffffffffu, sk, ps < 0 ? 0 : ps);
        if (ps >= 0) w = s0;
#pragma unroll 4
        for (int q = 0; q < t; ++q) {
            const double a = __shfl_sync(0xffffffffu, sk, q), c = __shfl_sync(0xffffffffu, ck, q);
            const double x = j > k ? a : hS[q * THREADS + tid], y = j > k ? hC[q * THREADS + tid] : c;
            const double v = fma(-x, y, w);
            w = q > ps ? v : w;
        }
        double sc = w * vkk;
        if (j == k) {
            sc = w = 0.0;
            ps = t;
            used = true;
            bj = bnew;
        } else {
            bj = fma(-bnew, w, bj);
            if (!used) dj = fma(-sc, w, dj);
        }
        hS[t * THREADS + tid] = sc;
        hC[t * THREADS + tid] = w;
        if (in) {
            p.S[(int64_t)t * n + j] = sc;
            p.C[(int64_t)t * n + j] = w;
        }
    }
    if (in) {
        p.used[j] = used;
        p.d[j] = dj;
        p.b[j] = bj;
        p.step[j] = (int8_t)ps;
    }
    if (rank == 0 && tid == 0) {
        p.st->count = t;
        if (t < p.tmax) {
            p.st->stop = 1;
            *p.deficit = -1;
        }
    }
    cl.sync();   // no CTA leaves while another may read its columns
}

// every element brought up to date with the block's pivots in their order;
// elements of a pivot row or column start from what its step left there
__global__ void __launch_bounds__(256) k_sqminl_update(int32_t n, double *V, const int8_t *step, const double *S,
                                                       const double *C, SqState *st) {
    __shared__ double ss[kPb][kTile + 2], cc[kPb][kTile + 2];
    __shared__ int8_t sr[kTile], sc[kTile];
    const int T = st->count;
    if (T <= 0) return;
    int bi, bj;
    tri_tile(blockIdx.x, bi, bj);
    const int r0 = bi * kTile, c0 = bj * kTile, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    for (int e = tid; e < T * kTile; e += 256) {
        const int q = e / kTile, i = e % kTile;
        cc[q][i] = r0 + i < n ? C[(int64_t)q * n + r0 + i] : 0.0;
        ss[q][i] = c0 + i < n ? S[(int64_t)q * n + c0 + i] : 0.0;
    }
    bool any = false;
    if (tid < kTile) {
        sr[tid] = r0 + tid < n ? step[r0 + tid] : -1;
        sc[tid] = c0 + tid < n ? step[c0 + tid] : -1;
        any = sr[tid] >= 0 || sc[tid] >= 0;
    }
    const bool pivots = __syncthreads_or(any);
    double w[4][4];
    int p0[4][4];
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int i = ty + 16 * a, jj = tx + 16 * b, r = r0 + i, c = c0 + jj;
            w[a][b] = 0.0;
            p0[a][b] = -1;
            if (r >= n || c > r) continue;
            if (pivots) {
                const int pr = sr[i], pc = sc[jj], q = max(pr, pc);
                p0[a][b] = q;
                if (q >= 0) {
                    w[a][b] = r == c ? -st->vkk[q] : S[(int64_t)q * n + (pr == q ? c : r)];
                    continue;
                }
            }
            w[a][b] = V[prow(r) + c];
        }
    if (!pivots) {
        for (int q = 0; q < T; ++q) {
            double x[4], y[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) { x[a] = -cc[q][ty + 16 * a]; y[a] = ss[q][tx + 16 * a]; }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) w[a][b] = fma(y[b], x[a], w[a][b]);
        }
    } else {
        for (int q = 0; q < T; ++q) {
            double x[4], y[4];
#pragma unroll
            for (int a = 0; a < 4; ++a) { x[a] = -cc[q][ty + 16 * a]; y[a] = ss[q][tx + 16 * a]; }
#pragma unroll
            for (int a = 0; a < 4; ++a)
#pragma unroll
                for (int b = 0; b < 4; ++b) {
                    const double v = fma(y[b], x[a], w[a][b]);
                    w[a][b] = q > p0[a][b] ? v : w[a][b];
                }
        }
    }
#pragma unroll
    for (int a = 0; a < 4; ++a)
#pragma unroll
        for (int b = 0; b < 4; ++b) {
            const int r = r0 + ty + 16 * a, c = c0 + tx + 16 * b;
            if (r < n && c <= r) V[prow(r) + c] = w[a][b];
        }
}

__global__ void k_sq_init(int32_t n, const double *V, double *d, int32_t *used, SqState *st, int32_t *deficit) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        d[i] = V[prow(i) + i];
        used[i] = 0;
    }
    if (i == 0) {
        st->count = st->stop = 0;
        *deficit = 0;
    }
}

// ------------------------------------------------------------ chdec2
// Rows i1-1 .. i0 (at most kPb) are the pivots of a block, from the last.
// First their own triangle, by four warps: lane c holds column i0 + c, warp w
// the rows 4 q + w of it in registers.  Row i is scaled by f_i = 1 / G(i, i)
// (the element itself where it is not positive, as chdec2 leaves it) and taken
// from the rows above: the next one at once, the others while the next pivot's
// reciprocal is under way.  The backward substitution of chslv2 uses the same
// rows in the same order and rides along.  Bound by the chain of pivots, some
// ten FP64 instructions of 64 clocks each: with one warp for all rows 37 us, now
// 22.
__device__ __forceinline__ void bar4(void) { asm volatile("bar.sync 1, 128;" ::: "memory"); }

__global__ void __launch_bounds__(128) k_chdec_diag(int32_t i0, int32_t nb, double *g, double *x, double *stat) {
    __shared__ double rowb[4][kPb], dv[kPb];
    const int c = threadIdx.x & 31, wq = threadIdx.x >> 5;
    double w[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) {
        const int r = 4 * q + wq;
        w[q] = (r < nb && c <= r) ? g[prow(i0 + r) + i0 + c] : 0.0;
    }
    double xc = c < nb ? x[i0 + c] : 0.0;
    double t = 0.0;
    const int top = nb - 1;
#pragma unroll
    for (int q = 0; q < 8; ++q)
        if (4 * q + wq == top) rowb[top & 3][c] = w[q];
#pragma unroll
    for (int i = kPb - 1; i >= 0; --i) {
        if (i >= nb) continue;
        bar4();
        const double *cur = rowb[i & 3], *prev = rowb[(i + 1) & 3];
        const double d = cur[i], wi = cur[c];
        const double f = d > 0x1p-120 && d < 0x1p120 ? newton_rcp(d) : (d > 0.0 ? 1.0 / d : d);
        if (threadIdx.x == 0) dv[i] = d;
        if (i + 1 < nb) {   // the pivot before, from the rows above this one
#pragma unroll
            for (int q = 0; q < 8; ++q)
                if (4 * q + wq < i) w[q] = fma(-t, prev[4 * q + wq], w[q]);   // used for c <= r
        }
        t = wi * f;   // (scaled element of column c)
        if (i > 0 && wq == ((i - 1) & 3)) {
            const int q = (i - 1) >> 2;
            w[q] = fma(-t, cur[i - 1], w[q]);
            rowb[(i - 1) & 3][c] = w[q];
        }
        const double xi = __shfl_sync(0xffffffffu, xc, i);
        if (c < i) xc = fma(-t, xi, xc);
        if (wq == (i & 3) && c <= i) g[prow(i0 + i) + i0 + c] = c < i ? t : f;
    }
    if (wq == 0) {
        if (c < nb) x[i0 + c] = xc;
        __syncwarp();
        // largest, smallest and number of the positive pivots
        const double d = c < nb ? dv[c] : 0.0, cnt = stat[2];
        const unsigned pos = __ballot_sync(0xffffffffu, d > 0.0);
        double hi = d > 0.0 ? d : 0.0, lo = d > 0.0 ? d : __longlong_as_double(0x7ff0000000000000ll);
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            hi = fmax(hi, __shfl_xor_sync(0xffffffffu, hi, o));
            lo = fmin(lo, __shfl_xor_sync(0xffffffffu, lo, o));
        }
        if (c == 0 && pos) {
            stat[0] = cnt == 0.0 ? hi : fmax(stat[0], hi);
            stat[1] = cnt == 0.0 ? lo : fmin(stat[1], lo);
            stat[2] = cnt + (double)__popc(pos);
        }
    }
}

// then the columns c < i0 of those rows, four lanes per column (lane s the rows
// 4 q + s): U the unscaled, R the scaled rows (also left in g); x of the
// columns.  FP64 instructions of single warps again: a thread per column took
// 35 us for 1,000 columns, now 11.
__global__ void __launch_bounds__(128) k_chdec_rows(int32_t i0, int32_t nb, double *g, double *x, double *U, double *R,
                                                    int64_t ld) {
    __shared__ double rat[kPb][kPb + 1], f[kPb], xb[kPb];
    const int tid = threadIdx.x, ln = tid & 31, sub = ln & 3, quad = ln & 28;
    const int64_t c = (int64_t)blockIdx.x * 32 + (tid >> 5) * 8 + (ln >> 2);
    const bool in = c < i0;
    double w[8];
#pragma unroll
    for (int q = 0; q < 8; ++q) w[q] = (in && 4 * q + sub < nb) ? g[prow(i0 + 4 * q + sub) + c] : 0.0;
    for (int e = tid; e < nb * nb; e += 128) {
        const int i = e / nb, r = e % nb;
        if (r <= i) {
            const double v = g[prow(i0 + i) + i0 + r];
            if (r < i) rat[i][r] = v;
            else f[i] = v;
        }
    }
    if (tid < nb) xb[tid] = x[i0 + tid];
    __syncthreads();
    double xs = 0.0;
#pragma unroll
    for (int i = kPb - 1; i >= 0; --i) {
        if (i >= nb) continue;
        const double u = __shfl_sync(0xffffffffu, w[i >> 2], quad | (i & 3));
#pragma unroll
        for (int q = 0; q <= i >> 2; ++q)
            if (q < i >> 2 || sub < (i & 3)) w[q] = fma(-u, rat[i][4 * q + sub], w[q]);
    }
#pragma unroll
    for (int q = 7; q >= 0; --q) {
        const int i = 4 * q + sub;
        if (i >= nb) continue;
        const double v = w[q] * f[i];
        if (in) {
            U[i * ld + c] = w[q];
            R[i * ld + c] = v;
            g[prow(i0 + i) + c] = v;
        }
        xs = fma(-v, xb[i], xs);
    }
    xs += __shfl_xor_sync(0xffffffffu, xs, 1);
    xs += __shfl_xor_sync(0xffffffffu, xs, 2);
    if (in && sub == 0) x[c] += xs;
}

// the leading i0 x i0 triangle: G(r, c) -= U(i, c) R(i, r), i from the last.
// Tiles of 32 x 32: the work of a tile of 64 (65,000 clocks) was the time of
// every launch with fewer tiles than SMs (61 us per block of 2,000 rows on
// average, now 46; FP64 floor 34).
constexpr int kCt = 32;
__global__ void __launch_bounds__(256) k_chdec_update(int32_t i0, int32_t nb, double *g, const double *U,
                                                      const double *R, int64_t ld) {
    __shared__ double su[kPb][kCt + 2], sr[kPb][kCt + 2];
    int bi, bj;
    tri_tile(blockIdx.x, bi, bj);
    const int r0 = bi * kCt, c0 = bj * kCt, tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    for (int e = tid; e < nb * kCt; e += 256) {
        const int q = e / kCt, i = e % kCt;
        sr[q][i] = r0 + i < i0 ? R[q * ld + r0 + i] : 0.0;
        su[q][i] = c0 + i < i0 ? U[q * ld + c0 + i] : 0.0;
    }
    double w[2][2];
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int r = r0 + ty + 16 * a, c = c0 + tx + 16 * b;
            w[a][b] = (r < i0 && c <= r) ? g[prow(r) + c] : 0.0;
        }
    __syncthreads();
#pragma unroll 4
    for (int q = nb - 1; q >= 0; --q) {
        double x[2], y[2];
#pragma unroll
        for (int a = 0; a < 2; ++a) { x[a] = -sr[q][ty + 16 * a]; y[a] = su[q][tx + 16 * a]; }
#pragma unroll
        for (int a = 0; a < 2; ++a)
#pragma unroll
            for (int b = 0; b < 2; ++b) w[a][b] = fma(y[b], x[a], w[a][b]);
    }
#pragma unroll
    for (int a = 0; a < 2; ++a)
#pragma unroll
        for (int b = 0; b < 2; ++b) {
            const int r = r0 + ty + 16 * a, c = c0 + tx + 16 * b;
            if (r < i0 && c <= r) g[prow(r) + c] = w[a][b];
        }
}

// ------------------------------------------------------------ chslv2, forward
// x(i) = x(i) G(i, i) - sum_{k < i} G(i, k) x(k).  Per block of kFb rows every
// CTA solves the block's triangle (one warp, two rows per lane) and takes it
// off its rows below; the solved block goes to out, as other CTAs still read
// x.
constexpr int kFb = 64;
__global__ void k_chslv_scale(int32_t n, const double *g, double *x) {
    const int64_t i = (int64_t)blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) x[i] *= g[prow(i) + i];
}
__global__ void __launch_bounds__(256) k_chslv_fwd(int32_t n, int32_t i0, const double *g, double *x, double *out) {
    __shared__ double t[kFb][kFb + 1], xs[kFb];
    const int tid = threadIdx.x, ln = tid & 31, wib = tid >> 5, nb = min(kFb, n - i0);
    for (int e = tid; e < nb * kFb; e += 256) {
        const int r = e / kFb, c = e % kFb;
        t[r][c] = c < r ? g[prow(i0 + r) + i0 + c] : 0.0;
    }
    __syncthreads();
    if (wib == 0) {
        double a = ln < nb ? x[i0 + ln] : 0.0, b = ln + 32 < nb ? x[i0 + ln + 32] : 0.0;
        for (int k = 0; k < nb; ++k) {
            const double xk = __shfl_sync(0xffffffffu, k < 32 ? a : b, k & 31);
            if (ln > k && ln < nb) a = fma(-t[ln][k], xk, a);
            if (ln + 32 > k && ln + 32 < nb) b = fma(-t[ln + 32][k], xk, b);
        }
        xs[ln] = a;
        xs[ln + 32] = b;
        if (blockIdx.x == 0) {
            if (ln < nb) out[i0 + ln] = a;
            if (ln + 32 < nb) out[i0 + ln + 32] = b;
        }
    }
    __syncthreads();
    for (int64_t r = i0 + kFb + (int64_t)blockIdx.x * 8 + wib; r < n; r += (int64_t)gridDim.x * 8) {
        const double *row = g + prow(r) + i0;
        double v = row[ln] * xs[ln] + row[ln + 32] * xs[ln + 32];
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (ln == 0) x[r] -= v;
    }
}

int64_t tiles_of(int64_t n, int tile) {
    const int64_t t = (n + tile - 1) / tile;
    return t * (t + 1) / 2;
}

}  // namespace

// S, C (or U, R): 2 kPb n; d or out: n; step: n bytes; state
int64_t packed_work_len(int32_t n) {
    return (2 * kPb + 1) * (int64_t)n + ((int64_t)n + 7) / 8 + (int64_t)(sizeof(SqState) + 7) / 8 + 8;
}

cudaError_t packed_sqminl(int32_t n, double *V, double *b, const double *diag, int32_t *used, int32_t *deficit,
                          double *work, cudaStream_t s) {
    SqParams p{};
    p.n = n;
    p.V = V;
    p.diag = diag;
    p.b = b;
    p.used = used;
    p.deficit = deficit;
    p.S = work;
    p.C = p.S + (int64_t)kPb * n;
    p.d = p.C + (int64_t)kPb * n;
    p.st = reinterpret_cast<SqState *>(p.d + n);
    p.step = reinterpret_cast<int8_t *>(p.st + 1);
    k_sq_init<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, V, p.d, used, p.st, deficit);
    // the panel's cluster: one row per thread where the rows allow it (128
    // threads per CTA, a warp per quarter of the SM; 256 above 2,048 rows), up to
    // 16 CTAs where the device takes such clusters, else 8; beyond that (4,096 or
    // 2,048 rows) the form with any number of rows per thread
    cudaLaunchConfig_t cfg{};
    cudaLaunchAttribute at{};
    at.id = cudaLaunchAttributeClusterDimension;
    at.val.clusterDim.y = at.val.clusterDim.z = 1;
    cfg.stream = s;
    cfg.attrs = &at;
    cfg.numAttrs = 1;
    // whether a cluster of 16 CTAs of this kernel can run
    auto takes16 = [&](auto *kern) {
        int nclust = 0;
        at.val.clusterDim.x = 16;
        cfg.gridDim = dim3(16);
        if (cudaFuncSetAttribute(kern, cudaFuncAttributeNonPortableClusterSizeAllowed, 1) == cudaSuccess &&
            cudaOccupancyMaxActiveClusters(&nclust, kern, &cfg) == cudaSuccess && nclust > 0)
            return true;
        cudaGetLastError();
        return false;
    };
    auto one_row = [&](auto *kern, int threads) {   // configures it when it fits
        cfg.blockDim = dim3(threads);
        cfg.dynamicSmemBytes = (size_t)2 * kPb * threads * sizeof(double);
        if (n > 16 * threads || cudaFuncSetAttribute(kern, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                                     (int)cfg.dynamicSmemBytes) != cudaSuccess) {
            cudaGetLastError();
            return false;
        }
        int cl = 1;
        while (cl * threads < n) cl *= 2;
        if (cl == 16 && !takes16(kern)) return false;
        at.val.clusterDim.x = cl;
        cfg.gridDim = dim3(cl);
        return true;
    };
    auto *kern = k_sqminl_panel_sm<128>;
    if (!one_row(kern, 128)) {
        kern = k_sqminl_panel_sm<256>;
        if (!one_row(kern, 256)) {
            kern = k_sqminl_panel;
            cfg.blockDim = dim3(kSqThreads);
            cfg.dynamicSmemBytes = 0;
            const int cl = takes16(kern) ? 16 : 8;
            at.val.clusterDim.x = cl;
            cfg.gridDim = dim3(cl);
        }
    }
    const unsigned nt = (unsigned)tiles_of(n, kTile);
    for (int32_t i = 0; i < n; i += kPb) {
        p.tmax = std::min(kPb, n - i);
        const cudaError_t e = cudaLaunchKernelEx(&cfg, kern, p);
        if (e != cudaSuccess) return e;
        k_sqminl_update<<<nt, 256, 0, s>>>(n, V, p.step, p.S, p.C, p.st);
    }
    return cudaGetLastError();
}

cudaError_t packed_chdec_solve(int32_t n, double *g, double *x, double *stat, double *work, cudaStream_t s) {
    double *U = work, *R = U + (int64_t)kPb * n, *out = R + (int64_t)kPb * n;
    for (int32_t i1 = n; i1 > 0; i1 -= kPb) {
        const int32_t i0 = std::max(0, i1 - kPb), nb = i1 - i0;
        k_chdec_diag<<<1, 128, 0, s>>>(i0, nb, g, x, stat);
        if (i0 == 0) break;
        k_chdec_rows<<<(unsigned)((i0 + 31) / 32), 128, 0, s>>>(i0, nb, g, x, U, R, n);
        k_chdec_update<<<(unsigned)tiles_of(i0, kCt), 256, 0, s>>>(i0, nb, g, U, R, n);
    }
    k_chslv_scale<<<(unsigned)((n + 255) / 256), 256, 0, s>>>(n, g, x);
    for (int32_t i0 = 0; i0 < n; i0 += kFb) {
        const int64_t rest = std::max<int64_t>(0, (int64_t)n - i0 - kFb);
        const unsigned gb = (unsigned)std::max<int64_t>(1, std::min<int64_t>((rest + 7) / 8, 304));
        k_chslv_fwd<<<gb, 256, 0, s>>>(n, i0, g, x, out);
    }
    cudaMemcpyAsync(x, out, sizeof(double) * n, cudaMemcpyDeviceToDevice, s);
    return cudaGetLastError();
}
