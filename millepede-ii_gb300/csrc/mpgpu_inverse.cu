// mpgpu_inverse.cu -- inverse of the QL-reduced global matrix from its
// blocked Cholesky factor: the dense form of the inversion that gives pede
// its parameter errors (minver, pede.f90:7838-7945, which inverts with
// sqminl, mpnum.f90:230-355).  With A = L L^T (mpgpu_dense.cu):
//   trtri  X = L^-1, in place, from the inverses of the diagonal blocks;
//   lauum  Z = X^T X (lower part), Z_ij = sum_{k >= i} X_ki^T X_kj.
// Both are lists of 128 x 128 tile products C = alpha sum_k A_k B_k^T +
// beta C run by one of two kernels: FP64 by exact slices on the tensor cores
// (mpgpu_ozaki.cu) or tcgen05 3xTF32 with FP32 accumulation in tensor memory
// over the whole K range (operands split once into TF32 hi/lo tiles).  Work:
// N^3/3 for each of trtri and lauum.
// trtri in FP64 doubles the inverted diagonal blocks: X_21 = -X_22 (L_21 X_11)
// for all pairs of blocks of b tiles at once, b = 4, 8, ... (blocks of four tiles
// come from the factorisation's super-blocks): eight products for 4,200 rows,
// the largest of 512 halves of tiles.  X_22 has the inverse unit of parameter k in
// column k and L_21 X_11 the unit in row k: the slices of these two are scaled by
// it.  In 3xTF32 it goes block
// column by block column from the last: for panel p, T = X_trail P (the panel P
// below the diagonal block times the already inverted trailing part), then
// X_panel = -T D_p with D_p = L_pp^-1.
// Measured in FP64, 4,200 rows: trtri 2.8 ms, lauum 1.6 ms (together 101 ms on
// the CUDA cores' FP64 units, trtri by panels).
#include <cuda_runtime.h>

#include <algorithm>
#include <vector>

#include "mpgpu_ctx.h"
#include "mpgpu_ozaki.h"
#include "mpgpu_tc.cuh"

namespace {

using tc::kNB;
using tc::kStageBytes;
using tc::kStages;
using tc::kTcSmem;
using tc::kTcThreads;
using tc::kOpBytes;
using tc::kTK;
constexpr int64_t kTileEl = (int64_t)kNB * kNB;

using tc::TileTask;

// ------------------------------------------------------------ tensor-core form
using tc::TcOp;

// Tiles rows [r0, r1) x columns [c0, c1) of the dense FP64 matrix M (or
// the tiles of M^T: tile (c, r) of the destination receives tile (r, c) of
// M transposed) split into TF32 hi + lo; the destination's tile column is
// the source's column less cOff (rows keep their index).
// A warp takes eight rows x 16 K: reads 128 bytes of each row (trans: 64 bytes
// of 16 rows), writes 512 contiguous bytes.  Four CTAs per tile: a CTA per tile
// with one element per thread at a time took 39 us for 156 tiles, now 24 (FP64
// conversions and the remainder: three instructions of 64 clocks per 32
// elements, 13 us).
constexpr int kSplitParts = 4;
__device__ __forceinline__ double widen(float f) {   // (double)f without the FP64 pipe
    const uint32_t b = __float_as_uint(f), e = (b >> 23) & 255u;
    if (e - 1u < 254u)
        return __hiloint2double((int)((b & 0x80000000u) | (((b & 0x7fffffffu) >> 3) + (896u << 20))), (int)(b << 29));
    return (double)f;
}
__global__ void __launch_bounds__(256) k_split_tiles(const double *M, int64_t ld, int32_t r0, int32_t r1, int32_t c0,
                                                     int32_t c1, int32_t trans, float *hi, float *lo, int64_t ntDst,
                                                     int32_t cOff) {
    const int64_t nc = c1 - c0, tile = blockIdx.x / kSplitParts;
    const int32_t tr = r0 + (int32_t)(tile / nc), tcc = c0 + (int32_t)(tile % nc);
    if (tr >= r1) return;
    const int64_t dst = trans ? ((int64_t)tcc * ntDst + tr) * kTileEl
                              : ((int64_t)tr * ntDst + (tcc - cOff)) * kTileEl;
    const int ln = threadIdx.x & 31, wib = threadIdx.x >> 5, r7 = ln & 7, k4 = ln >> 3;
    constexpr int kItems = 128 / kSplitParts;   // 8 chunks x 16 row groups
    const int part = (int)(blockIdx.x % kSplitParts) * kItems;
#pragma unroll
    for (int i = 0; i < kItems / 8; ++i) {
        const int it = part + i * 8 + wib, u = (it & 15) * 8 + r7, k = (it >> 4) * kTK + k4 * 4;
        double x[4];
        if (!trans) {
            const double2 *p = reinterpret_cast<const double2 *>(M + ((int64_t)tr * kNB + u) * ld + (int64_t)tcc * kNB + k);
            const double2 v = p[0], w = p[1];
            x[0] = v.x; x[1] = v.y; x[2] = w.x; x[3] = w.y;
        } else {
            const double *p = M + ((int64_t)tr * kNB + k) * ld + (int64_t)tcc * kNB + u;
#pragma unroll
            for (int q = 0; q < 4; ++q) x[q] = p[q * ld];
        }
        uint32_t h[4], l[4];
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(h[q]) : "f"((float)x[q]));
            const double rest = x[q] - widen(__uint_as_float(h[q]));
            asm("cvt.rna.tf32.f32 %0, %1;" : "=r"(l[q]) : "f"((float)rest));
        }
        const int64_t o = dst + (it >> 4) * (kNB * kTK) + ((it & 15) * 4 + k4) * 32 + r7 * 4;
        *reinterpret_cast<uint4 *>(hi + o) = make_uint4(h[0], h[1], h[2], h[3]);
        *reinterpret_cast<uint4 *>(lo + o) = make_uint4(l[0], l[1], l[2], l[3]);
    }
}

// One CTA per task: the K range of the task streamed chunk by chunk (16
// columns of one K tile per chunk) through three stages by a producer thread,
// hi*hi + hi*lo + lo*hi accumulated in one FP32 tensor-memory accumulator over
// all chunks, then C = alpha acc + beta C in FP64 (coalesced through shared
// memory; alpha +-1, beta 0 or 1).  Bounded mbarrier waits: a wait that runs out
// sets *err = -1 and the CTA finishes without writing C.  Without a task list
// the CTAs take the lower triangle of tiles from tile (trail0, trail0) on, each
// with K tiles [0, trailK) of rows i and j: the trailing update of a block
// column.  Two CTAs per SM, so that one's epilogue (one FP64 addition per
// element, 8,200 clocks) runs beside the other's products (6 instructions of 64
// clocks per chunk); 32 KB per chunk from L2.  With the copies issued by all
// threads and three FP64 instructions per element a trailing update of 11,175
// tiles with K = 512 took 5.0 ms, now 2.2 (beside the panels).
__global__ void __launch_bounds__(kTcThreads, 2) k_tile_gemm_tc(TcOp A, TcOp B, double *C, int64_t ldc,
                                                                const TileTask *tasks, int32_t trail0, int32_t trailK,
                                                                double alpha, double beta, int32_t *err) {
    extern __shared__ __align__(128) char tsm[];
    __shared__ uint64_t full[kStages], empty[kStages], done;
    __shared__ uint32_t tbase;
    const int tid = threadIdx.x, wib = tid >> 5, ln = tid & 31;
    TileTask t;
    if (tasks) {
        t = tasks[blockIdx.x];
    } else {
        const int64_t q = blockIdx.x;
        int bi = (int)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
        while ((int64_t)bi * (bi + 1) / 2 > q) bi--;
        while ((int64_t)(bi + 1) * (bi + 2) / 2 <= q) bi++;
        const int bj = (int)(q - (int64_t)bi * (bi + 1) / 2);
        t = TileTask{trail0 + bi, trail0 + bj, 0, trailK, trail0 + bi, trail0 + bj};
    }
    const int per = kNB / kTK;   // chunks per K tile
    const int nch = (t.k1 - t.k0) * per;
    if (nch <= 0) return;
    const uint32_t sbase = (tc::smem_u32(tsm) + 127u) & ~127u;
    if (wib == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc::smem_u32(&tbase)),
                     "r"(kNB));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (tid == 0) {
        for (int st = 0; st < kStages; ++st) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(tc::smem_u32(&full[st])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(tc::smem_u32(&empty[st])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(tc::smem_u32(&done)));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tbase;
    bool ok = true;
    int issued = 0;   // producer: chunks whose copies were issued; MMA warp: chunks committed
    if (wib == 4) {
        if (ln == 0) {
            for (int c = 0; c < nch; ++c) {
                const int st = c % kStages;
                if (c >= kStages && !tc::mbar_wait(tc::smem_u32(&empty[st]), ((c / kStages) - 1) & 1)) {
                    ok = false;
                    break;
                }
                const int64_t k = t.k0 + c / per, in = (int64_t)(c % per) * (kNB * kTK);
                const int64_t ta = ((int64_t)t.aRow * A.nt + k) * kTileEl + in;
                const int64_t tb = ((int64_t)t.bRow * B.nt + k) * kTileEl + in;
                const uint32_t bar = tc::smem_u32(&full[st]), s0 = sbase + st * kStageBytes;
                asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(kStageBytes)
                             : "memory");
                tc::bulk_load(s0, A.hi + ta, kOpBytes, bar);
                tc::bulk_load(s0 + kOpBytes, A.lo + ta, kOpBytes, bar);
                tc::bulk_load(s0 + 2 * kOpBytes, B.hi + tb, kOpBytes, bar);
                tc::bulk_load(s0 + 3 * kOpBytes, B.lo + tb, kOpBytes, bar);
                issued = c + 1;
            }
            // the last chunks' copies have landed (also after a failed wait)
            for (int d = issued > kStages ? issued - kStages : 0; d < issued; ++d)
                if (!tc::mbar_wait(tc::smem_u32(&full[d % kStages]), (d / kStages) & 1)) ok = false;
        }
    } else if (wib == 5) {
        if (ln == 0) {
            for (int c = 0; c < nch; ++c) {
                const int st = c % kStages;
                if (!tc::mbar_wait(tc::smem_u32(&full[st]), (c / kStages) & 1)) {
                    ok = false;
                    break;
                }
                asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                const uint32_t sb = sbase + st * kStageBytes;
#pragma unroll
                for (int kk = 0; kk < kTK / 8; ++kk) {
                    const uint32_t off = kk * 256;   // 8 tf32 = 2 core matrices along K
                    const uint64_t dah = tc::umma_desc(sb + off), dal = tc::umma_desc(sb + kOpBytes + off);
                    const uint64_t dbh = tc::umma_desc(sb + 2 * kOpBytes + off), dbl = tc::umma_desc(sb + 3 * kOpBytes + off);
                    tc::mma_tf32(tmem, dah, dbh, (c > 0 || kk > 0) ? 1u : 0u);
                    tc::mma_tf32(tmem, dah, dbl, 1u);
                    tc::mma_tf32(tmem, dal, dbh, 1u);
                }
                tc::commit_to(tc::smem_u32(&empty[st]));
                issued = c + 1;
            }
            if (ok) tc::commit_to(tc::smem_u32(&done));
            // the MMAs issued are done (also after a failed wait)
            for (int d = issued > kStages ? issued - kStages : 0; d < issued; ++d)
                if (!tc::mbar_wait(tc::smem_u32(&empty[d % kStages]), (d / kStages) & 1)) ok = false;
        }
    } else {
        ok = tc::mbar_wait_warp(tc::smem_u32(&done), 0);
        asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
        if (ok) {
            // all MMAs are done, so that the stages are free
            float *epi = reinterpret_cast<float *>(tsm + (sbase - tc::smem_u32(tsm))) + wib * 32 * 33;
            const int64_t rowBase = (int64_t)t.cRow * kNB + wib * 32;
            const int64_t colBase = (int64_t)t.cCol * kNB;
            const uint32_t flip = alpha < 0.0 ? 0x80000000u : 0u;
            for (int cb = 0; cb < kNB / 32; ++cb) {
                double *cp = C + rowBase * ldc + colBase + cb * 32 + ln;
                uint32_t v[32];
                tc::tmem_ld32(tmem + ((uint32_t)(wib * 32) << 16) + (uint32_t)(cb * 32), v);
#pragma unroll
                for (int q = 0; q < 32; ++q) epi[ln * 33 + q] = __uint_as_float(v[q] ^ flip);
                __syncwarp();
#pragma unroll 1
                for (int r0 = 0; r0 < 32; r0 += 16) {
                    double cv[16];
#pragma unroll
                    for (int r = 0; r < 16; ++r) cv[r] = beta != 0.0 ? cp[(r0 + r) * ldc] : 0.0;
#pragma unroll
                    for (int r = 0; r < 16; ++r) {
                        const double x = widen(epi[(r0 + r) * 33 + ln]);
                        cp[(r0 + r) * ldc] = beta != 0.0 ? cv[r] + x : x;
                    }
                }
                __syncwarp();
            }
        }
    }
    if (!ok) atomicExch(err, -1);
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (wib == 0)
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(kNB));
}

// diagonal block p of X: D_p = L_pp^-1 from its transposed copy
// (DinvT[p][r][c] = D_p[c][r]), zero above the diagonal
__global__ void k_set_diag_inverse(double *L, int64_t ld, int32_t p, const double *DinvT) {
    const double *D = DinvT + (int64_t)p * kTileEl;
    for (int e = blockIdx.x * blockDim.x + threadIdx.x; e < kTileEl; e += gridDim.x * blockDim.x) {
        const int i = e / kNB, j = e % kNB;
        L[((int64_t)p * kNB + i) * ld + (int64_t)p * kNB + j] = j <= i ? D[(int64_t)j * kNB + i] : 0.0;
    }
}

// the inverted blocks of four tiles (XS: rows of 4 kNB columns, zero above the
// diagonal) to the tiles on and below the diagonal; eight rows per CTA
__global__ void __launch_bounds__(256) k_set_super_inverse(double *L, int64_t ld, const double *XS) {
    const int64_t r0 = (int64_t)blockIdx.x * 8, c0 = r0 / (4 * kNB) * (4 * kNB);
    const int cols = (int)((r0 / kNB + 1) * kNB - c0);
    for (int e = threadIdx.x; e < 8 * cols; e += 256) {
        const int64_t r = r0 + e / cols;
        L[r * ld + c0 + e % cols] = XS[r * 4 * kNB + e % cols];
    }
}

// a CTA per row in turn (a square root per element to find its row took 217 us
// for 4,200 rows, now 31; 141 MB)
__global__ void __launch_bounds__(256) k_dense_lower_to_packed(const double *Z, int64_t ld, int64_t n, double *Zp) {
    for (int64_t i = blockIdx.x; i < n; i += gridDim.x) {
        const double *z = Z + i * ld;
        double *o = Zp + i * (i + 1) / 2;
#pragma unroll 4
        for (int64_t j = threadIdx.x; j <= i; j += 256) o[j] = z[j];
    }
}

}  // namespace

// L (npad x npad, dense row-major, the lower Cholesky factor with the
// inverses of its diagonal blocks in DinvT and of its blocks of four tiles in
// XS, and the exponents of its rows' units in kexp) is replaced by X = L^-1; Z =
// X^T X (lower part) is written to Zd and its leading n x n block packed
// into Zp.  mode 0: FP64 tile products by slices; mode 1: tensor-core 3xTF32.
int32_t dense_inverse_device(mpgpu_ctx *c, double *L, int64_t npad, int64_t n, int mode, const double *DinvT,
                             const double *XS, const int32_t *kexp, double *Zd, double *Zp, int32_t *dErr) {
    cudaStream_t s = c->stream;
    const int32_t np = (int32_t)(npad / kNB);
    const int64_t ld = npad;
    // tasks of every trtri step (mode 0: T = L_21 X_11, then X_21 = -X_22 T,
    // for every block size; mode 1: T products, then the panel scaling) and of
    // lauum
    std::vector<TileTask> tk;
    std::vector<int64_t> stepT(np + 2), stepS(np + 2);
    if (mode == 0) {
        int lv = 0;
        for (int32_t b = 4; b < np; b *= 2, ++lv)
            for (int sec = 0; sec < 2; ++sec) {
                (sec ? stepS : stepT)[lv] = (int64_t)tk.size();
                std::vector<TileTask> t;
                for (int32_t base = 0; base + b < np; base += 2 * b)
                    for (int32_t i = base + b; i < std::min(base + 2 * b, np); ++i)
                        for (int32_t j = base; j < base + b; ++j)
                            t.push_back(sec ? TileTask{i, j, base + b, i + 1, i, j} : TileTask{i, j, j, base + b, i, j});
                std::stable_sort(t.begin(), t.end(),
                                 [](const TileTask &a, const TileTask &b) { return a.k1 - a.k0 > b.k1 - b.k0; });
                tk.insert(tk.end(), t.begin(), t.end());
            }
        stepT[lv] = (int64_t)tk.size();
    } else {
        for (int32_t p = np - 1; p >= 0; --p) {
            stepT[p] = (int64_t)tk.size();
            for (int32_t r = p + 1; r < np; ++r) tk.push_back({r, p, p + 1, r + 1, r - p - 1, 0});
            stepS[p] = (int64_t)tk.size();
            for (int32_t r = p + 1; r < np; ++r) tk.push_back({r - p - 1, 0, 0, 1, r, p});
        }
    }
    const int64_t lauum0 = (int64_t)tk.size();
    {
        // longest K first
        std::vector<TileTask> la;
        for (int32_t i = 0; i < np; ++i)
            for (int32_t j = 0; j <= i; ++j) la.push_back({i, j, i, np, i, j});
        std::stable_sort(la.begin(), la.end(),
                         [](const TileTask &a, const TileTask &b) { return a.k1 - a.k0 > b.k1 - b.k0; });
        tk.insert(tk.end(), la.begin(), la.end());
    }
    TileTask *dTask = nullptr;
    double *T = nullptr;
    float *xhi = nullptr, *xlo = nullptr, *thi = nullptr, *tlo = nullptr, *phi = nullptr, *plo = nullptr,
          *dhi = nullptr, *dlo = nullptr;
    // mode 0: slices of the two operands, W tiles of every row at a time
    uint8_t *img[2] = {nullptr, nullptr};
    int32_t *ex[2] = {nullptr, nullptr};
    auto release = [&] {
        for (int q = 0; q < 2; ++q) {
            cudaFree(img[q]);
            cudaFree(ex[q]);
        }
        cudaFree(dTask); cudaFree(T);
        cudaFree(xhi); cudaFree(xlo); cudaFree(thi); cudaFree(tlo); cudaFree(phi); cudaFree(plo);
        cudaFree(dhi); cudaFree(dlo);
    };
    cudaError_t e = cudaMalloc(&dTask, sizeof(TileTask) * tk.size());
    const int64_t full = (int64_t)np * np * kTileEl;
    if (mode == 1) {
        if (e == cudaSuccess) e = cudaMalloc(&T, sizeof(double) * npad * kNB);
        // X (non-transposed) and L^T, later X^T, split tile by tile; the
        // panel T and the diagonal inverse D_p split per step
        if (e == cudaSuccess) e = cudaMalloc(&xhi, sizeof(float) * full);
        if (e == cudaSuccess) e = cudaMalloc(&xlo, sizeof(float) * full);
        if (e == cudaSuccess) e = cudaMalloc(&phi, sizeof(float) * full);
        if (e == cudaSuccess) e = cudaMalloc(&plo, sizeof(float) * full);
        if (e == cudaSuccess) e = cudaMalloc(&thi, sizeof(float) * (int64_t)np * kTileEl);
        if (e == cudaSuccess) e = cudaMalloc(&tlo, sizeof(float) * (int64_t)np * kTileEl);
        if (e == cudaSuccess) e = cudaMalloc(&dhi, sizeof(float) * kTileEl);
        if (e == cudaSuccess) e = cudaMalloc(&dlo, sizeof(float) * kTileEl);
    }
    // W: all K tiles up to 64 (C is read and written once per W tiles, 64 of
    // them take 400 us), fewer where the memory does not suffice
    int32_t W = c->lean ? 4 : std::min(64, (np + 3) / 4 * 4);
    oz::Op oa{}, ob{};
    if (mode == 0 && e == cudaSuccess) {
        for (;; W = std::max(4, W / 8 * 4)) {
            const size_t bytes = (size_t)np * W * oz::kTileBytes;
            e = cudaMalloc(&img[0], bytes);
            if (e == cudaSuccess) e = cudaMalloc(&img[1], bytes);
            if (e == cudaSuccess || W == 4) break;
            cudaGetLastError();
            for (uint8_t *&p : img) {
                cudaFree(p);
                p = nullptr;
            }
        }
        for (int q = 0; q < 2; ++q)
            if (e == cudaSuccess) e = cudaMalloc(&ex[q], sizeof(int32_t) * np * (W / 4) * kNB);
        oa = oz::Op{img[0], ex[0], W, W / 4};
        ob = oz::Op{img[1], ex[1], W, W / 4};
    }
    if (e == cudaSuccess)
        e = cudaMemcpyAsync(dTask, tk.data(), sizeof(TileTask) * tk.size(), cudaMemcpyHostToDevice, s);
    if (e != cudaSuccess) { release(); return cuda_err(c, e, "blocked inverse workspace"); }
    if (mode == 1) {
        MPG_CUDA(c, smem_optin((const void *)k_tile_gemm_tc));
        // L^T tiles (p, k) for k > p: the panels of the original factor
        for (int32_t p = 0; p < np - 1; ++p)
            k_split_tiles<<<kSplitParts * (np - 1 - p), 256, 0, s>>>(L, ld, p + 1, np, p, p + 1, 1, phi, plo, np, 0);
    }
    MPG_CUDA(c, cudaMemsetAsync(dErr, 0, sizeof(int32_t), s));
    // launches of mode 0 release the workspace when they fail
#define MPG_OZ(call)                                                        \
    do {                                                                    \
        const cudaError_t oe_ = (call);                                     \
        if (oe_ != cudaSuccess) {                                           \
            release();                                                      \
            return cuda_err(c, oe_, #call);                                 \
        }                                                                   \
    } while (0)
    const int64_t nla = (int64_t)np * (np + 1) / 2;
    if (mode == 0) {
        // ---- trtri: T in Zd, which lauum fills afterwards
        k_set_super_inverse<<<(unsigned)np * 16, 256, 0, s>>>(L, ld, XS);
        int lv = 0;
        for (int32_t b = 4; b < np; b *= 2, ++lv) {
            const int32_t pairs = (np - b + 2 * b - 1) / (2 * b);
            for (int32_t w0 = 0; w0 < b; w0 += W) {
                const int32_t w1 = std::min(w0 + W, b);
                MPG_OZ(oz_split(L, ld, b, 2 * b, w0, w1, 0, 0, oa, 0, w0, 2, s, pairs, 2 * b, np));
                MPG_OZ(oz_split(L, ld, 0, b, w0, w1, 1, 2, ob, 0, w0, 2, s, pairs, 2 * b, np));
                MPG_OZ(oz_tile_gemm(oa, ob, Zd, ld, dTask + stepT[lv], stepS[lv] - stepT[lv], 0, 0, 2, 1.0, 0.0, dErr,
                                    s, oz::Window{2 * b, w0, w1 - w0}));
            }
            for (int32_t w0 = b; w0 < 2 * b; w0 += W) {
                const int32_t w1 = std::min(w0 + W, 2 * b);
                MPG_OZ(oz_split(L, ld, b, 2 * b, w0, w1, 0, 1, oa, 0, w0, 2, s, pairs, 2 * b, np, 0, kexp, 1));
                MPG_OZ(oz_split(Zd, ld, 0, b, w0, w1, 1, 0, ob, 0, w0, 2, s, pairs, 2 * b, np, 0, kexp, -1));
                MPG_OZ(oz_tile_gemm(oa, ob, L, ld, dTask + stepS[lv], stepT[lv + 1] - stepS[lv], 0, 0, 2, -1.0, 0.0,
                                    dErr, s, oz::Window{2 * b, w0, w1 - w0}));
            }
        }
        // ---- lauum
        for (int32_t w0 = 0; w0 < np; w0 += W) {
            const int32_t w1 = std::min(w0 + W, np);
            MPG_OZ(oz_split(L, ld, 0, np, w0, w1, 1, 2, oa, 0, w0, 2, s));
            MPG_OZ(oz_tile_gemm(oa, oa, Zd, ld, dTask + lauum0, nla, 0, 0, 2, 1.0, 0.0, dErr, s,
                                oz::Window{0, w0, w1 - w0}));
        }
    } else {
        // ---- trtri, panels from the last
        for (int32_t p = np - 1; p >= 0; --p) {
            const int32_t m = np - 1 - p;
            if (m > 0) {
                k_tile_gemm_tc<<<m, kTcThreads, kTcSmem, s>>>(TcOp{xhi, xlo, np}, TcOp{phi, plo, np}, T, kNB,
                                                              dTask + stepT[p], 0, 0, 1.0, 0.0, dErr);
                k_split_tiles<<<kSplitParts * m, 256, 0, s>>>(T, kNB, 0, m, 0, 1, 0, thi, tlo, 1, 0);
                k_split_tiles<<<kSplitParts, 256, 0, s>>>(DinvT + (int64_t)p * kTileEl, kNB, 0, 1, 0, 1, 0, dhi, dlo, 1, 0);
                k_tile_gemm_tc<<<m, kTcThreads, kTcSmem, s>>>(TcOp{thi, tlo, 1}, TcOp{dhi, dlo, 1}, L, ld,
                                                              dTask + stepS[p], 0, 0, -1.0, 0.0, dErr);
            }
            k_set_diag_inverse<<<16, 256, 0, s>>>(L, ld, p, DinvT);
            // the finished column of X, split for the later steps' products
            k_split_tiles<<<kSplitParts * (m + 1), 256, 0, s>>>(L, ld, p, np, p, p + 1, 0, xhi, xlo, np, 0);
            MPG_CUDA(c, cudaGetLastError());
        }
        // ---- lauum: X^T tiles (i, k) for k >= i (into the L^T area)
        for (int32_t i = 0; i < np; ++i)
            k_split_tiles<<<kSplitParts * (np - i), 256, 0, s>>>(L, ld, i, np, i, i + 1, 1, phi, plo, np, 0);
        k_tile_gemm_tc<<<(unsigned)nla, kTcThreads, kTcSmem, s>>>(TcOp{phi, plo, np}, TcOp{phi, plo, np}, Zd, ld,
                                                                  dTask + lauum0, 0, 0, 1.0, 0.0, dErr);
    }
#undef MPG_OZ
    MPG_CUDA(c, cudaGetLastError());
    k_dense_lower_to_packed<<<4096, 256, 0, s>>>(Zd, ld, n, Zp);
    int32_t h = 0;
    e = cudaMemcpyAsync(&h, dErr, sizeof(int32_t), cudaMemcpyDeviceToHost, s);
    if (e == cudaSuccess) e = cudaStreamSynchronize(s);
    release();
    if (e != cudaSuccess) return cuda_err(c, e, "blocked inverse");
    if (h < 0) return set_err(c, MPGPU_ERR_TIMEOUT, "tensor-core tile product: barrier wait ran out");
    return MPGPU_OK;
}

// Launchers for the blocked Cholesky (mpgpu_dense.cu).
cudaError_t tc_split_tiles(const double *M, int64_t ld, int32_t r0, int32_t r1, int32_t c0, int32_t c1, float *hi,
                           float *lo, int64_t ntDst, int32_t cOff, cudaStream_t s) {
    const int64_t n = (int64_t)(r1 - r0) * (c1 - c0);
    if (n <= 0) return cudaSuccess;
    k_split_tiles<<<(unsigned)(kSplitParts * n), 256, 0, s>>>(M, ld, r0, r1, c0, c1, 0, hi, lo, ntDst, cOff);
    return cudaGetLastError();
}

cudaError_t tc_tile_gemm(const TcOp &A, const TcOp &B, double *C, int64_t ldc, const TileTask *tasks, int64_t ntask,
                         int32_t trail0, int32_t trailK, double alpha, double beta, int32_t *err, cudaStream_t s) {
    if (ntask <= 0) return cudaSuccess;
    cudaError_t e = smem_optin((const void *)k_tile_gemm_tc);
    if (e != cudaSuccess) return e;
    k_tile_gemm_tc<<<(unsigned)ntask, kTcThreads, kTcSmem, s>>>(A, B, C, ldc, tasks, trail0, trailK, alpha, beta, err);
    return cudaGetLastError();
}
