// mpgpu_ozaki.h -- FP64 tile products on the tensor cores by exact slices
// (mpgpu_ozaki.cu).
#pragma once
#include <cuda_runtime.h>
#include <stdint.h>

#include "mpgpu_tc.cuh"

namespace oz {

constexpr int kSlices = 8;                          // 7-bit digits per value
constexpr int kImages = kSlices + 4;                // the digits, and digits 4..7 times 2^-7
constexpr int64_t kTileBytes = 128 * 128 * 2 * kImages;   // one sliced 128 x 128 tile
constexpr int kGroupTiles = 4;                      // most K tiles of one scale group (K = 512)

// Sliced operand: tile (r, k) at img + (r * nt + k) * kTileBytes, the
// exponents of row i of tile row r for scale group g at ex[(r * ng + g) * 128 +
// i]; group of K tile k: k >> gs.
struct Op {
    uint8_t *img;
    int32_t *ex;
    int64_t nt, ng;
};

// K tiles of a product: those of a task within [off, off + width), off = (cRow
// / lvl) lvl + add (lvl 0: add); the operands hold tile off + k at k.  A task
// that began before the window adds to C.
struct Window {
    int32_t lvl = 0, add = 0, width = 1 << 28;
};

}  // namespace oz

// Slices row tiles [r0, r1) and K tiles [k0, k1) of the dense FP64 matrix M
// into tile (r - rOff, k - cOff) of dst (scale group (k - cOff) >> gs); trans:
// tile (r, k) is taken from tile (k, r) of M transposed; tri 1: only k <= r, 2:
// only k >= r.  count > 1: the same for r0, r1, k0, k1 and cOff moved by step, 2
// step, ... tiles; tiles from lim on are left out.  wrap > 0: M holds column
// tile c at c mod wrap (the K tiles of a group then wrap at most at its ends).
// kexp: K value k (counted over all K tiles, not wrapped) is taken times 2^(ksign
// kexp[k]); the other operand takes the opposite sign.
cudaError_t oz_split(const double *M, int64_t ld, int32_t r0, int32_t r1, int32_t k0, int32_t k1, int trans, int tri,
                     const oz::Op &dst, int32_t rOff, int32_t cOff, int gs, cudaStream_t s, int32_t count = 1,
                     int32_t step = 0, int32_t lim = 1 << 28, int32_t wrap = 0, const int32_t *kexp = nullptr,
                     int ksign = 1);
// C(cRow, cCol) = alpha sum_k A(aRow, k) B(bRow, k)^T + beta C over a device
// task list, or (tasks null) over the lower triangle of tiles from tile
// (trail0, trail0) on with K tiles [0, trailK) (tc_tile_gemm's convention).
// alpha +-1, beta 0 or 1.
cudaError_t oz_tile_gemm(const oz::Op &A, const oz::Op &B, double *C, int64_t ldc, const tc::TileTask *tasks,
                         int64_t ntask, int32_t trail0, int32_t trailK, int gs, double alpha, double beta,
                         int32_t *err, cudaStream_t s, const oz::Window &win = {});
