// mpgpu_ozaki.cu -- FP64 tile products C = alpha A B^T + beta C on the tcgen05
// tensor cores by error-free slices (the scheme of Ozaki, Ogita, Oishi & Rump
// 2012, with the operands' rows scaled to fixed point).
//
// GB300's FP64 units give 2 multiply-adds per SM and clock (0.63 T/s), its
// bf16 tensor cores some 4,000.  Every operand row is scaled by a power of two
// over a group of at most 512 K values, rounded to 56-bit fixed point and cut
// into eight balanced 7-bit digits, which bf16 holds exactly.  The products of
// digits i and j with i + j = d share one FP32 accumulator: at most 8 pairs x
// 512 K x 2^12 = 2^24, so every sum is exact in FP32.  The eight accumulators
// of a tile (digits i + j <= 7, 36 products) are combined in 64-bit integers
// and added to C in FP64 once per group.  The seven products with i + j = 8 are
// added to the last accumulator, one digit of each taken from a copy scaled by
// 2^-7 (FP32 holds that sum to far below its unit): without them the error was
// up to 3.7 times that of an FP64 sum where rows have a few large elements
// (and the digits' squares gave the diagonal a bias).  What is left out or
// rounded is below 2^-56 of (row maximum of A) x (row maximum of B) per term,
// of either sign, against 2^-53 of the partial sums in FP64.  That is as good
// as an FP64 sum where the elements of a row are of like size, as they are in a
// Cholesky factor, whose row k has the unit of parameter k (over factors of the
// barrel and telescope matrices 5 to 100 times below the FP64 sum's error) and
// in its inverse's columns.  Where the unit runs along K (a row of the inverse
// times a column of a product of the factor) both operands are scaled by powers
// of two per K value, which cancel in the product: without, the error grew by the
// ratio of the units (relative errors of the inverse of 1,024 rows 2e-13 for
// units 2e4 apart, 2e-9 for 1e8; with the scales as for equal units).
//
// Per chunk of 16 K a CTA multiplies 128 x 16 by 16 x 64 in 43 instructions
// from 70 KB of shared memory (three stages, filled by bulk copies of images
// that oz_split lays out in the tensor cores' core-matrix order), its
// accumulators fill the 512 columns of tensor memory.  Bounds: operand reads
// of the 64-column instructions (6 KB of shared memory each), then the
// epilogue (some 100 integer instructions per element and group) and 70 KB per chunk
// from L2.  Measured: X^T X of 33 x 33 triangular tiles (561 tiles, 12 K tiles
// on average) 1.20 ms, three quarters of it the instructions (54 clocks each),
// one seventh the epilogue (with eight warps for it 1.31 ms; with C read and
// written once per group and the integers converted by FP64 instructions, by
// four warps, 1.50 ms).
#include <cuda_runtime.h>

#include <algorithm>

#include "mpgpu_ctx.h"
#include "mpgpu_ozaki.h"

namespace {

using oz::kImages;
using oz::kSlices;
using oz::kTileBytes;
using oz::Op;
constexpr int kNB = tc::kNB;
constexpr int kChunkK = 16;                          // K per stage
constexpr int kChunks = kNB / kChunkK;               // per K tile
constexpr int kSliceBytes = kNB * kChunkK * 2;       // 4 KB: a slice's chunk image
constexpr int kChunkBytes = kImages * kSliceBytes;   // 48 KB: a tile's chunk, all slices
constexpr int kN = 64;                               // columns of C per CTA
constexpr int kImagesB = kImages - 1;                // B needs no scaled digit 4
constexpr int kStageBytes = kChunkBytes + kImagesB * (kSliceBytes / 2);
constexpr int kStages = 3;
constexpr int kSmem = kStages * kStageBytes + 128;
constexpr int kEpi = 16;                             // epilogue warps
constexpr int kThreads = 32 * (kEpi + 2);            // and producer, MMA issuer
constexpr int kNanEx = 1 << 28;                      // row with an infinity or NaN

// K-major core matrices of 8 rows x 16 bytes: 128 bytes apart along K, 256
// along the rows
__device__ __forceinline__ uint64_t desc16(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(128 >> 4) << 16) | ((uint64_t)(256 >> 4) << 32) |
           (1ull << 46);
}

// D f32, A and B bf16, K-major, N = 64, M = 128
constexpr uint32_t kIdescBf16 =
    (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(kN >> 3) << 17) | ((uint32_t)(kNB >> 4) << 24);

// KEEP: what the tensor core does with its copy of A's tile: 0 fetch A, 1 fetch
// and keep it, 2 use the kept one, 3 use it for the last time
template <int KEEP>
__device__ __forceinline__ void mma_bf16(uint32_t tmem, uint64_t ad, uint64_t bd, uint32_t acc) {
#define MPG_MMA(KIND)                                                            \
    asm volatile("{\n.reg .pred p;\nsetp.ne.b32 p, %4, 0;\n"                     \
                 "tcgen05.mma.cta_group::1.kind::f16" KIND " [%0], %1, %2, %3, p;\n}\n" ::"r"(tmem), \
                 "l"(ad), "l"(bd), "r"(kIdescBf16), "r"(acc))
    if (KEEP == 1) MPG_MMA(".collector::a::fill");
    else if (KEEP == 2) MPG_MMA(".collector::a::use");
    else if (KEEP == 3) MPG_MMA(".collector::a::lastuse");
    else MPG_MMA("");
#undef MPG_MMA
}

using tc::bulk_load;
using tc::commit_to;

// eight columns of four accumulators, kN columns apart, and the wait for them
__device__ __forceinline__ void tmem_ld4x8(uint32_t t, uint32_t (&r)[4][8]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%32];\n"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%8,%9,%10,%11,%12,%13,%14,%15}, [%33];\n"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%16,%17,%18,%19,%20,%21,%22,%23}, [%34];\n"
        "tcgen05.ld.sync.aligned.32x32b.x8.b32 {%24,%25,%26,%27,%28,%29,%30,%31}, [%35];\n"
        "tcgen05.wait::ld.sync.aligned;\n"
        : "=r"(r[0][0]), "=r"(r[0][1]), "=r"(r[0][2]), "=r"(r[0][3]), "=r"(r[0][4]), "=r"(r[0][5]), "=r"(r[0][6]),
          "=r"(r[0][7]), "=r"(r[1][0]), "=r"(r[1][1]), "=r"(r[1][2]), "=r"(r[1][3]), "=r"(r[1][4]), "=r"(r[1][5]),
          "=r"(r[1][6]), "=r"(r[1][7]), "=r"(r[2][0]), "=r"(r[2][1]), "=r"(r[2][2]), "=r"(r[2][3]), "=r"(r[2][4]),
          "=r"(r[2][5]), "=r"(r[2][6]), "=r"(r[2][7]), "=r"(r[3][0]), "=r"(r[3][1]), "=r"(r[3][2]), "=r"(r[3][3]),
          "=r"(r[3][4]), "=r"(r[3][5]), "=r"(r[3][6]), "=r"(r[3][7])
        : "r"(t), "r"(t + kN), "r"(t + 2 * kN), "r"(t + 3 * kN)
        : "memory");
}

// (hi 2^28 + lo) 2^e rounded to nearest, |hi| and |lo| below 2^46.  In integers,
// as the two conversions and the product took three FP64 instructions (64
// clocks of a quarter of the SM each).
__device__ __forceinline__ double combine(long long hi, long long lo, int e) {
    long long h = hi + (lo >> 28);
    uint32_t l = (uint32_t)lo & 0xfffffffu;
    const long long sign = h & (long long)0x8000000000000000ull;
    if (h < 0) {   // the magnitude
        h = l ? ~h : -h;
        l = (0u - l) & 0xfffffffu;
    }
    const unsigned long long u = (unsigned long long)h;
    if (u == 0) return scalbn(sign ? -(double)l : (double)l, e);
    const int z = __clzll((long long)u);   // 17..63
    const unsigned long long ll = (unsigned long long)l << 36;
    const unsigned long long w = (u << z) | (ll >> (64 - z));
    const unsigned long long rest = ll << z;
    unsigned long long m = w >> 11;   // 53 bits
    const uint32_t low = (uint32_t)w & 0x7ffu;
    m += (low > 0x400u || (low == 0x400u && ((m & 1) || rest != 0))) ? 1 : 0;
    const int f = 1023 + 91 - z + e;   // exponent field of 2^63 2^(28 - z) 2^e
    if (f > 0 && f < 2046) return __longlong_as_double(sign | (long long)(((unsigned long long)(f - 1) << 52) + m));
    return scalbn(__longlong_as_double(sign | (long long)((1022ull << 52) + m)), f - 1023);
}

__global__ void __launch_bounds__(kThreads, 1) k_oz_gemm(Op A, Op B, double *C, int64_t ldc, const tc::TileTask *tasks,
                                                         int32_t trail0, int32_t trailK, int gs, double alpha,
                                                         double beta, int32_t *err, oz::Window win) {
    extern __shared__ __align__(128) char osm[];
    __shared__ uint64_t full[kStages], empty[kStages], accFull, accEmpty;
    __shared__ uint32_t tbase;
    const int tid = threadIdx.x, wib = tid >> 5, ln = tid & 31;
    const int half = blockIdx.x & 1;
    tc::TileTask t;
    if (tasks) {
        t = tasks[blockIdx.x >> 1];
    } else {
        const int64_t q = blockIdx.x >> 1;
        int bi = (int)((sqrt(8.0 * (double)q + 1.0) - 1.0) * 0.5);
        while ((int64_t)bi * (bi + 1) / 2 > q) bi--;
        while ((int64_t)(bi + 1) * (bi + 2) / 2 <= q) bi++;
        const int bj = (int)(q - (int64_t)bi * (bi + 1) / 2);
        t = tc::TileTask{trail0 + bi, trail0 + bj, 0, trailK, trail0 + bi, trail0 + bj};
    }
    const int kOff = (win.lvl > 0 ? t.cRow / win.lvl * win.lvl : 0) + win.add;
    const bool began = t.k0 < kOff;
    t.k0 = max(t.k0 - kOff, 0);
    t.k1 = min(t.k1 - kOff, win.width);
    if (t.k1 <= t.k0) return;
    if (wib == 0) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;\n" ::"r"(tc::smem_u32(&tbase)),
                     "r"(512));
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;\n");
    }
    if (tid == 0) {
        for (int st = 0; st < kStages; ++st) {
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(tc::smem_u32(&full[st])));
            asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(tc::smem_u32(&empty[st])));
        }
        asm volatile("mbarrier.init.shared::cta.b64 [%0], 1;\n" ::"r"(tc::smem_u32(&accFull)));
        asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;\n" ::"r"(tc::smem_u32(&accEmpty)), "n"(32 * kEpi));
        asm volatile("fence.mbarrier_init.release.cluster;\n" ::: "memory");
    }
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    const uint32_t tmem = tbase;
    const uint32_t sbase = (tc::smem_u32(osm) + 127u) & ~127u;
    bool ok = true;
    // waits that run out leave *err = -1; every role then leaves its loop, and
    // the copies and MMAs already issued are waited for (bounded) below
    int issued = 0;   // producer: chunks whose copies were issued; MMA warp: chunks committed
    if (wib == kEpi) {
        if (ln == 0) {
            int c = 0;
            for (int k = t.k0; k < t.k1 && ok; ++k) {
                const uint8_t *a = A.img + ((int64_t)t.aRow * A.nt + k) * kTileBytes;
                const uint8_t *b = B.img + ((int64_t)t.bRow * B.nt + k) * kTileBytes + half * (kSliceBytes / 2);
                for (int q = 0; q < kChunks; ++q, ++c) {
                    const int st = c % kStages;
                    if (c >= kStages && !tc::mbar_wait(tc::smem_u32(&empty[st]), ((c / kStages) - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    const uint32_t bar = tc::smem_u32(&full[st]), s0 = sbase + st * kStageBytes;
                    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n" ::"r"(bar), "r"(kStageBytes)
                                 : "memory");
                    bulk_load(s0, a + (int64_t)q * kChunkBytes, kChunkBytes, bar);
#pragma unroll
                    for (int j = 0; j < kImagesB; ++j)
                        bulk_load(s0 + kChunkBytes + j * (kSliceBytes / 2),
                                  b + (int64_t)q * kChunkBytes + (j < kSlices ? j : j + 1) * kSliceBytes, kSliceBytes / 2,
                                  bar);
                    issued = c + 1;
                }
            }
            // the last chunks' copies have landed (also after a failed wait)
            for (int d = issued > kStages ? issued - kStages : 0; d < issued; ++d)
                if (!tc::mbar_wait(tc::smem_u32(&full[d % kStages]), (d / kStages) & 1)) ok = false;
        }
    } else if (wib == kEpi + 1) {
        if (ln == 0) {
            int c = 0, grp = 0;
            for (int k = t.k0; k < t.k1 && ok; ++k) {
                const bool first = k == t.k0 || (k >> gs) != ((k - 1) >> gs);
                const bool last = k == t.k1 - 1 || (k >> gs) != ((k + 1) >> gs);
                if (first && grp > 0) {
                    if (!tc::mbar_wait(tc::smem_u32(&accEmpty), (grp - 1) & 1)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                }
                for (int q = 0; q < kChunks; ++q, ++c) {
                    const int st = c % kStages;
                    if (!tc::mbar_wait(tc::smem_u32(&full[st]), (c / kStages) & 1)) {
                        ok = false;
                        break;
                    }
                    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
                    const uint32_t sa = sbase + st * kStageBytes, sb = sa + kChunkBytes;
#pragma unroll
                    for (int i = 0; i < kSlices; ++i) {
                        // digit i of A with all the digits of B that it meets, so
                        // that its tile is fetched once; digits 1..3 also with the
                        // scaled copy of B's digit 8 - i
                        const uint64_t ad = desc16(sa + i * kSliceBytes);
                        const int n = kSlices - i + (i > 0 && i < 4);
#pragma unroll
                        for (int j = 0; j < n; ++j) {
                            const int d = j < kSlices - i ? i + j : kSlices - 1;            // accumulator
                            const int im = j < kSlices - i ? j : kSlices - i + 3;           // image of B
                            const uint64_t bd = desc16(sb + im * (kSliceBytes / 2));
                            const uint32_t acc = (first && q == 0 && i == 0) ? 0u : 1u;
                            if (n == 1) mma_bf16<0>(tmem + (uint32_t)(d * kN), ad, bd, acc);
                            else if (j == 0) mma_bf16<1>(tmem + (uint32_t)(d * kN), ad, bd, acc);
                            else if (j < n - 1) mma_bf16<2>(tmem + (uint32_t)(d * kN), ad, bd, acc);
                            else mma_bf16<3>(tmem + (uint32_t)(d * kN), ad, bd, acc);
                        }
                    }
#pragma unroll
                    for (int i = 4; i < kSlices; ++i)   // scaled digits 4..7 of A with digits 4..1 of B
                        mma_bf16<0>(tmem + (uint32_t)((kSlices - 1) * kN), desc16(sa + (i + 4) * kSliceBytes),
                                    desc16(sb + (kSlices - i) * (kSliceBytes / 2)), 1u);
                    commit_to(tc::smem_u32(&empty[st]));
                    issued = c + 1;
                }
                if (ok && last) {
                    commit_to(tc::smem_u32(&accFull));
                    ++grp;
                }
            }
            for (int d = issued > kStages ? issued - kStages : 0; d < issued; ++d)
                if (!tc::mbar_wait(tc::smem_u32(&empty[d % kStages]), (d / kStages) & 1)) ok = false;
        }
    } else {
        // warps w, w + 4, ... take kC columns each of the rows of tensor memory
        // that they can read; C stays in registers over the groups
        constexpr int kC = kN / (kEpi / 4);
        const int rw = (wib & 3) * 32, c0 = (wib >> 2) * kC;
        const int64_t row = (int64_t)t.cRow * kNB + rw + ln;
        double *cp = C + row * ldc + (int64_t)t.cCol * kNB + half * kN + c0;
        double c[kC];
        const bool add = began || beta != 0.0;
#pragma unroll
        for (int q = 0; q < kC; q += 2) {
            const double2 v = add ? *reinterpret_cast<const double2 *>(cp + q) : make_double2(0.0, 0.0);
            c[q] = v.x;
            c[q + 1] = v.y;
        }
        int grp = 0;
        for (int k = t.k0; k < t.k1; ++k) {
            if (!(k == t.k1 - 1 || (k >> gs) != ((k + 1) >> gs))) continue;
            const int64_t g = k >> gs;
            const int er = A.ex[((int64_t)t.aRow * A.ng + g) * kNB + rw + ln];
            const int el = B.ex[((int64_t)t.bRow * B.ng + g) * kNB + half * kN + c0 + ln % kC];   // lane = column
            if (!tc::mbar_wait_warp(tc::smem_u32(&accFull), grp & 1)) {
                ok = false;
                break;
            }
            asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
#pragma unroll
            for (int cb = 0; cb < kC / 8; ++cb) {
                const uint32_t tc0 = tmem + ((uint32_t)rw << 16) + (uint32_t)(c0 + cb * 8);
                uint32_t vh[4][8], vl[4][8];
                tmem_ld4x8(tc0, vh);
                tmem_ld4x8(tc0 + 4 * kN, vl);
#pragma unroll
                for (int q = 0; q < 8; ++q) {
                    long long hi = 0, lo = 0;
#pragma unroll
                    for (int d = 0; d < 4; ++d) {
                        hi = (hi << 7) + (long long)__float2int_rn(__uint_as_float(vh[d][q]));
                        lo = (lo << 7) + (long long)__float2int_rn(__uint_as_float(vl[d][q]));
                    }
                    const int ec = __shfl_sync(0xffffffffu, el, cb * 8 + q);
                    double x = combine(hi, lo, er + ec - 61);
                    if (er == kNanEx || ec == kNanEx) x = __longlong_as_double(0x7ff8000000000000ll);
                    c[cb * 8 + q] += alpha < 0.0 ? -x : x;
                }
            }
            asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
            asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];\n" ::"r"(tc::smem_u32(&accEmpty)) : "memory");
            ++grp;
        }
        if (ok)
#pragma unroll
            for (int q = 0; q < kC; q += 2) *reinterpret_cast<double2 *>(cp + q) = make_double2(c[q], c[q + 1]);
    }
    if (!ok) atomicExch(err, -1);
    __syncwarp();
    asm volatile("tcgen05.fence::before_thread_sync;\n" ::: "memory");
    __syncthreads();
    asm volatile("tcgen05.fence::after_thread_sync;\n" ::: "memory");
    if (wib == 0) asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;\n" ::"r"(tmem), "r"(512));
}

// One CTA per 32 rows and scale group (a CTA per row tile left most SMs idle: 40
// us per launch in the inversion of 4,200 rows, now 14): the row maxima's
// exponents over the group's K tiles, then every eight consecutive K values of
// a row as 16-byte pieces, one per slice, in core-matrix order (eight rows of a
// piece are 128 contiguous bytes).  Integer arithmetic on the bit patterns
// throughout.  KS: the K values are scaled by powers of two, kexp[k] (or -kexp[k])
// added to their exponents.
constexpr int kSplitRows = 32;
constexpr int kZeroEx = -(1 << 20);   // exponent of zero in scaled rows
template <bool KS>
__global__ void __launch_bounds__(256) k_oz_split(const double *M, int64_t ld, int32_t r0, int32_t k0, int32_t k1,
                                                  int trans, int tri, Op dst, int32_t rOff, int32_t cOff, int gs,
                                                  int32_t step, int32_t lim, int32_t wrap, const int32_t *kexp,
                                                  int ksign) {
    __shared__ int emax[kSplitRows];
    const int tid = threadIdx.x, ln = tid & 31, wib = tid >> 5;
    r0 += blockIdx.z * step;
    k0 += blockIdx.z * step;
    k1 = min(k1 + (int32_t)blockIdx.z * step, lim);
    cOff += blockIdx.z * step;
    const int32_t R = r0 + blockIdx.x / (kNB / kSplitRows), Rd = R - rOff;
    const int h0 = (blockIdx.x % (kNB / kSplitRows)) * kSplitRows;   // first row in the tile
    {
        const int32_t g0 = ((((k0 - cOff) >> gs) + (int32_t)blockIdx.y) << gs) + cOff;
        k1 = min(k1, g0 + (1 << gs));
        k0 = max(k0, g0);
        if (tri == 1) k1 = min(k1, R + 1);
        if (tri == 2) k0 = max(k0, R);
        if (k0 >= k1 || R >= lim) return;
    }
    const int K = (k1 - k0) * kNB;
    // first row and K value in M
    const int64_t row0 = (int64_t)(trans && wrap > 0 ? R % wrap : R) * kNB + h0;
    const int64_t kk0 = (int64_t)(!trans && wrap > 0 ? k0 % wrap : k0) * kNB;
    const int32_t *ke = KS ? kexp + (int64_t)k0 * kNB : nullptr;
    if (tid < kSplitRows) emax[tid] = KS ? kZeroEx : 0;
    __syncthreads();
    // exponent field of K value q of a row, scaled
    auto field = [&](double x, int q) {
        const int f = (int)((__double_as_longlong(x) >> 52) & 0x7ff);
        if (!KS) return f;
        return f == 2047 ? kNanEx : x == 0.0 ? kZeroEx : max(f, 1) + ksign * __ldg(ke + q);
    };
    if (!trans) {
        for (int r = wib; r < kSplitRows; r += 8) {
            const double2 *p = reinterpret_cast<const double2 *>(M + (row0 + r) * ld + kk0);
            int e = KS ? kZeroEx : 0;
#pragma unroll 4
            for (int q = ln; q < K / 2; q += 32) {
                const double2 v = p[q];
                e = max(e, max(field(v.x, 2 * q), field(v.y, 2 * q + 1)));
            }
#pragma unroll
            for (int o = 16; o > 0; o >>= 1) e = max(e, __shfl_xor_sync(0xffffffffu, e, o));
            if (ln == 0) emax[r] = e;
        }
    } else {
        const double *p = M + kk0 * ld + row0 + ln;
        int e = KS ? kZeroEx : 0;
#pragma unroll 8
        for (int q = wib; q < K; q += 8) e = max(e, field(p[(int64_t)q * ld], q));
        atomicMax(&emax[ln], e);
    }
    __syncthreads();
    if (tid < kSplitRows)
        dst.ex[((int64_t)Rd * dst.ng + ((k0 - cOff) >> gs)) * kNB + h0 + tid] =
            KS ? (emax[tid] == kNanEx ? kNanEx : emax[tid] - 1022)
               : (emax[tid] == 2047 ? kNanEx : max(emax[tid], 1) - 1022);
    uint8_t *out = dst.img + ((int64_t)Rd * dst.nt + (k0 - cOff)) * kTileBytes;
    const int nk8 = K / 8, total = kSplitRows * nk8;
    for (int it = tid; it < total; it += 256) {
        // a warp writes 4 x 128 contiguous bytes per slice; it reads 64 bytes of
        // each of 8 rows x 4 pieces, or (trans) 64 bytes of 32 columns
        const int r7 = it & 7, k8 = (it >> 3) % nk8, rl = ((it >> 3) / nk8) * 8 + r7, rg = h0 / 8 + (it >> 3) / nk8;
        double x[8];
        if (!trans) {
            const double2 *p = reinterpret_cast<const double2 *>(M + (row0 + rl) * ld + kk0 + k8 * 8);
#pragma unroll
            for (int q = 0; q < 4; ++q) {
                const double2 v = p[q];
                x[2 * q] = v.x;
                x[2 * q + 1] = v.y;
            }
        } else {
            const double *p = M + (kk0 + k8 * 8) * ld + row0 + rl;
#pragma unroll
            for (int q = 0; q < 8; ++q) x[q] = p[(int64_t)q * ld];
        }
        uint32_t w[kImages][4];
        const int em = KS ? emax[rl] : max(emax[rl], 1);
#pragma unroll
        for (int q = 0; q < 8; ++q) {
            const long long b = __double_as_longlong(x[q]);
            const int e = max((int)((b >> 52) & 0x7ff), 1) + (KS ? ksign * __ldg(ke + k8 * 8 + q) : 0);
            long long m = b & 0xfffffffffffffll;
            if ((b >> 52) & 0x7ff) m |= 0x10000000000000ll;
            // x 2^(55 - exponent), |.| < 2^55, rounded to an integer (a zero has
            // no part in the scaled maximum)
            const int sh = KS && m == 0 ? 0 : em - e - 2;
            if (sh <= 0) m <<= -sh;
            else m = sh > 60 ? 0 : (m + (1ll << (sh - 1))) >> sh;
            if (b < 0) m = -m;
#pragma unroll
            for (int sl = kSlices - 1; sl >= 0; --sl) {
                int d;
                if (sl > 0) {
                    d = (int)((m + 64) & 127) - 64;
                    m = (m - d) >> 7;
                } else {
                    d = (int)m;
                }
                const float f = (float)d;
                const uint32_t h = __float_as_uint(f) >> 16;   // exact in bf16
                if (q & 1) w[sl][q >> 1] |= h << 16;
                else w[sl][q >> 1] = h;
                if (sl >= 4) {
                    const uint32_t hs = __float_as_uint(f * 0.0078125f) >> 16;
                    if (q & 1) w[sl + 4][q >> 1] |= hs << 16;
                    else w[sl + 4][q >> 1] = hs;
                }
            }
        }
        const int k = k8 * 8;
        uint8_t *o = out + (int64_t)(k / kNB) * kTileBytes + (int64_t)((k % kNB) / kChunkK) * kChunkBytes +
                     (rg * (kChunkK / 8) + ((k % kChunkK) >> 3)) * 128 + r7 * 16;
#pragma unroll
        for (int sl = 0; sl < kImages; ++sl)
            *reinterpret_cast<uint4 *>(o + sl * kSliceBytes) = make_uint4(w[sl][0], w[sl][1], w[sl][2], w[sl][3]);
    }
}

}  // namespace

cudaError_t oz_split(const double *M, int64_t ld, int32_t r0, int32_t r1, int32_t k0, int32_t k1, int trans, int tri,
                     const oz::Op &dst, int32_t rOff, int32_t cOff, int gs, cudaStream_t s, int32_t count, int32_t step,
                     int32_t lim, int32_t wrap, const int32_t *kexp, int ksign) {
    if (r1 <= r0 || k1 <= k0 || count <= 0) return cudaSuccess;
    const int ng = ((k1 - 1 - cOff) >> gs) - ((k0 - cOff) >> gs) + 1;
    const dim3 grid((unsigned)((r1 - r0) * (kNB / kSplitRows)), (unsigned)ng, (unsigned)count);
    (kexp ? k_oz_split<true> : k_oz_split<false>)<<<grid, 256, 0, s>>>(M, ld, r0, k0, k1, trans, tri, dst, rOff, cOff, gs,
                                                                       step, lim, wrap, kexp, ksign);
    return cudaGetLastError();
}

cudaError_t oz_tile_gemm(const oz::Op &A, const oz::Op &B, double *C, int64_t ldc, const tc::TileTask *tasks,
                         int64_t ntask, int32_t trail0, int32_t trailK, int gs, double alpha, double beta,
                         int32_t *err, cudaStream_t s, const oz::Window &win) {
    if (ntask <= 0) return cudaSuccess;
    const cudaError_t e = smem_optin((const void *)k_oz_gemm);
    if (e != cudaSuccess) return e;
    k_oz_gemm<<<(unsigned)(2 * ntask), kThreads, kSmem, s>>>(A, B, C, ldc, tasks, trail0, trailK, gs, alpha, beta, err,
                                                             win);
    return cudaGetLastError();
}
