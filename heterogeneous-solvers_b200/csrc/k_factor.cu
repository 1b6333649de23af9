// k_factor.cu — kernels of the blocked right-looking Cholesky in FP64:
// diagonal-block POTRF, panel TRSM and the SYRK/GEMM trailing update.
//
// Reference kernels replaced (paths relative to the reference root):
//   MatrixOperations.cpp:7-191          cholesky / cholesky_GPU / cholesky_optimizedGPU
//   MatrixMatrixOperations.cpp:5-144    triangularSolve{,_optimizedGPU,_optimizedCPU}
//   MatrixMatrixOperations.cpp:146-361  symmetricMatrixMatrixDiagonal{,...}
//   MatrixMatrixOperations.cpp:364-906  matrixMatrixStep{,...}
//
// The trailing update is the only O(N^3) part.  For bsz a multiple of 128 it
// runs on the FP64 tensor pipe (DMMA, mma.sync m8n8k4 f64): 128x64 output tiles,
// two CTAs an SM, K streamed in 16-wide slabs through a 3-stage cp.async ring in
// shared memory, accumulators held in registers and initialised with -C so the
// result is C - sum_k a_ik b_jk accumulated in k order (the factor's large updates are
// k_split_update.cu's).  Other block sizes use
// a scalar fallback with the reference's accumulation order.  The diagonal block
// of bsz 128 and 256 is k_diag.cu's.
#include "hs_gp.cuh"
#include "hs_internal.cuh"
#include "hs_mixed.cuh"

namespace hs {
namespace {

// ------------------------------------------------------------------ POTRF
// In-shared-memory POTRF of an n x n (n <= 128) sub-block with leading
// dimension ld: the reference's column-by-column right-looking order
// (MatrixOperations.cpp:23-57), rows >= valid untouched, strict upper triangle
// of valid rows zeroed.  A pivot that is not > 0 on a valid row records its
// global row in *info.
__global__ void __launch_bounds__(512) potrf_smem_kernel(double* __restrict__ Ablk, int ld, int n, int valid,
                                                         long long* __restrict__ info, long long row_base) {
    extern __shared__ double S[];
    const int sld = n + 1;
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e % n;
        S[i * sld + j] = Ablk[(size_t)i * ld + j];
    }
    __syncthreads();
    for (int k = 0; k < n; ++k) {
        const double piv = S[k * sld + k];
        const double s = sqrt(piv);
        if (threadIdx.x == 0 && k < valid && !(piv > 0.0)) atomicMin(info, row_base + k);
        for (int i = k + 1 + (int)threadIdx.x; i < valid; i += blockDim.x) S[i * sld + k] = S[i * sld + k] / s;
        __syncthreads();
        if (threadIdx.x == 0) S[k * sld + k] = s;
        // lower trailing part: j in (k, n), i in [j, valid); one warp per column,
        // lanes over rows (no index divisions, no idle lanes above the diagonal)
        {
            const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, nw = blockDim.x >> 5;
            for (int j = k + 1 + warp; j < valid; j += nw) {
                const double sjk = S[j * sld + k];
                for (int i = j + lane; i < valid; i += 32) S[i * sld + j] = S[i * sld + j] - S[i * sld + k] * sjk;
            }
        }
        __syncthreads();
    }
    for (int e = threadIdx.x; e < n * n; e += blockDim.x) {
        const int i = e / n, j = e % n;
        if (i >= valid) continue;
        Ablk[(size_t)i * ld + j] = (j > i) ? 0.0 : S[i * sld + j];
    }
    // the reference also writes a_kk = sqrt(a_kk) on padding rows (MatrixOperations.cpp:38-40)
    for (int k = valid + (int)threadIdx.x; k < n; k += blockDim.x) Ablk[(size_t)k * ld + k] = S[k * sld + k];
}

// global-memory fallback (bsz > 256): one CTA, same order as the reference
__global__ void __launch_bounds__(1024) potrf_global_kernel(double* __restrict__ B, int n, int valid,
                                                            long long* __restrict__ info, long long row_base) {
    for (int k = 0; k < n; ++k) {
        const double piv = B[(size_t)k * n + k];
        const double s = sqrt(piv);
        if (threadIdx.x == 0 && k < valid && !(piv > 0.0)) atomicMin(info, row_base + k);
        __syncthreads();
        for (int i = k + 1 + (int)threadIdx.x; i < valid; i += blockDim.x) B[(size_t)i * n + k] /= s;
        __syncthreads();
        if (threadIdx.x == 0) B[(size_t)k * n + k] = s;
        const int m = n - k - 1;
        for (int64_t e = threadIdx.x; e < (int64_t)m * m; e += blockDim.x) {
            const int j = k + 1 + (int)(e / m);
            const int i = k + 1 + (int)(e % m);
            if (i >= j && i < valid) B[(size_t)i * n + j] -= B[(size_t)i * n + k] * B[(size_t)j * n + k];
        }
        __syncthreads();
    }
    for (int64_t e = threadIdx.x; e < (int64_t)n * n; e += blockDim.x) {
        const int i = (int)(e / n), j = (int)(e % n);
        if (i < valid && j > i) B[e] = 0.0;
    }
}

// ------------------------------------------------------------------ TRSM
// B <- B L^-T for slabs of up to 64 rows: each CTA keeps its slab in shared
// memory and walks the columns in 32-wide chunks: solve the chunk against the
// chunk's diagonal triangle (column order, divisions as the reference's CPU
// kernel, MatrixMatrixOperations.cpp:125-139), then subtract the chunk's
// contribution from the columns to its right, accumulating in k order.
constexpr int kTrsmRows = 64;
constexpr int kTrsmCh = 32;

struct TrsmArgs {
    const double* L;   // triangle (lower), leading dimension ldL
    int ldL;
    int n;             // triangle size = columns of B
    double* A;         // base for B items
    int ldB;
    int64_t item0;     // first B block id
    int slabs;         // slabs per B item
    int rows_last;     // rows in each item
    int64_t block_elems;  // stride between B blocks (elements)
};

__global__ void __launch_bounds__(256) trsm_kernel(TrsmArgs a) {
    extern __shared__ double sm[];
    const int n = a.n;
    const int bld = n + 1;
    double* Bs = sm;                                  // kTrsmRows x (n+1)
    double* Tc = Bs + kTrsmRows * bld;                // kTrsmCh x (kTrsmCh+1)
    double* Lp = Tc + kTrsmCh * (kTrsmCh + 1);        // n x (kTrsmCh+1)
    const int item = blockIdx.x / a.slabs;
    const int slab = blockIdx.x % a.slabs;
    const double* Lt = a.L;
    double* B = a.A + (size_t)(a.item0 + item) * a.block_elems + (size_t)slab * kTrsmRows * a.ldB;
    const int rows = min(kTrsmRows, a.rows_last - slab * kTrsmRows);
    for (int e = threadIdx.x; e < rows * n; e += blockDim.x) {
        const int r = e / n, c = e % n;
        Bs[r * bld + c] = B[(size_t)r * a.ldB + c];
    }
    const int nch = (n + kTrsmCh - 1) / kTrsmCh;
    for (int ch = 0; ch < nch; ++ch) {
        const int k0 = ch * kTrsmCh;
        const int kn = min(kTrsmCh, n - k0);
        const int rest = n - (k0 + kn);
        __syncthreads();
        for (int e = threadIdx.x; e < kn * kn; e += blockDim.x) {
            const int i = e / kn, k = e % kn;
            Tc[i * (kTrsmCh + 1) + k] = Lt[(size_t)(k0 + i) * a.ldL + (k0 + k)];
        }
        for (int e = threadIdx.x; e < rest * kn; e += blockDim.x) {
            const int i = e / kn, k = e % kn;
            Lp[i * (kTrsmCh + 1) + k] = Lt[(size_t)(k0 + kn + i) * a.ldL + (k0 + k)];
        }
        __syncthreads();
        // chunk solve: one thread per row (rows are independent)
        for (int r = threadIdx.x; r < rows; r += blockDim.x) {
            double* row = Bs + r * bld + k0;
            for (int k = 0; k < kn; ++k) {
                const double bk = row[k] / Tc[k * (kTrsmCh + 1) + k];
                row[k] = bk;
                for (int i = k + 1; i < kn; ++i) row[i] = row[i] - Tc[i * (kTrsmCh + 1) + k] * bk;
            }
        }
        __syncthreads();
        // trailing columns: b_rc -= sum_k b_rk * L[c][k], k ascending
        for (int e = threadIdx.x; e < rows * rest; e += blockDim.x) {
            const int r = e / rest, c = e % rest;
            double v = Bs[r * bld + k0 + kn + c];
            const double* bk = Bs + r * bld + k0;
            const double* lc = Lp + c * (kTrsmCh + 1);
            for (int k = 0; k < kn; ++k) v = v - lc[k] * bk[k];
            Bs[r * bld + k0 + kn + c] = v;
        }
    }
    __syncthreads();
    for (int e = threadIdx.x; e < rows * n; e += blockDim.x) {
        const int r = e / n, c = e % n;
        B[(size_t)r * a.ldB + c] = Bs[r * bld + c];
    }
}

size_t trsm_smem(int n) {
    return (size_t)(kTrsmRows * (n + 1) + kTrsmCh * (kTrsmCh + 1) + n * (kTrsmCh + 1)) * sizeof(double);
}

// ------------------------------------------------------------------ DMMA tile
constexpr int BK = 16, SPAD = 20;

__device__ __forceinline__ void cp_async16(void* smem, const void* gmem) {
    const unsigned s = static_cast<unsigned>(__cvta_generic_to_shared(smem));
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;\n" ::"r"(s), "l"(gmem));
}
__device__ __forceinline__ void cp_async_commit() { asm volatile("cp.async.commit_group;\n" ::); }
template <int N>
__device__ __forceinline__ void cp_async_wait() { asm volatile("cp.async.wait_group %0;\n" ::"n"(N)); }

// A CTA computes a TM x TN output tile with (TM/WM) x (TN/WN) warps of WM x WN
// (m8n8k4 sub-tiles), K streamed in 16-wide slabs through an ST-stage cp.async
// ring with rows padded to SPAD doubles (row stride 40 banks: the eight rows a
// fragment load touches fall in distinct bank groups).
template <int TM, int TN, int WM, int WN, int ST>
struct DTile {
    static constexpr int kWarpsN = TN / WN;
    static constexpr int kThreads = 32 * (TM / WM) * (TN / WN);
    static constexpr int kMi = WM / 8, kNi = WN / 8;
    static constexpr int kBRow = TN + 4;  // PRODUCT: B k-major, rows of 4 k 32 bytes apart modulo 128
    static constexpr int kBStage = TN * SPAD > BK * kBRow ? TN * SPAD : BK * kBRow;
    static constexpr int kSmem = ST * (TM * SPAD + kBStage) * (int)sizeof(double);
    static constexpr int kChunks = (TM + TN) * (BK / 2);  // 16-byte copies a stage
    static_assert(kChunks % kThreads == 0, "copies must split evenly over the threads");
    static_assert((TM * (BK / 2)) % 32 == 0, "A and B copies must not share a warp");
};

// PRODUCT = 0: C (TM x TN, ldc) <- C - A (TM x K, lda) B (TN x K, ldb)^T,
//   accumulated from -C in k order; with `lower`, entry (r, c) is written only
//   if c + shift <= r (a tile that crosses the diagonal of a diagonal block).
// PRODUCT = 2: C <- A B^T with B (TN x K, ldb) upper triangular (B[c][k] = 0 for k < c):
//   a warp skips the K slabs before its first column.  C may be A itself.
// PRODUCT = 1: C <- A B with B (K x TN, ldb) upper triangular (B[k][c] = 0 for
//   k > c): a warp skips the K slabs past its last column, and what B holds below its
//   WN x WN diagonal blocks is not used.  C may be A itself: every load of A completes
//   before the first store.
template <int TM, int TN, int WM, int WN, int ST, int PRODUCT>
__device__ __forceinline__ void dmma_tile_t(double* C, int64_t ldc, const double* Ag, int64_t lda,
                                            const double* __restrict__ Bg, int64_t ldb, int K, bool lower, int shift,
                                            double* smem) {
    using D = DTile<TM, TN, WM, WN, ST>;
    double* As = smem;                   // [ST][TM][SPAD]
    double* Bs = smem + ST * TM * SPAD;  // [ST][TN][SPAD]
    const int tid = threadIdx.x;
    const int warp = tid >> 5, lane = tid & 31;
    // PRODUCT: columns have sums of different lengths; warps w and w + 4 share a scheduler, so the
    // second four take the columns in reverse
    const int wm = warp / D::kWarpsN;
    const int wn = PRODUCT && warp >= 4 ? D::kWarpsN - 1 - warp % 4 % D::kWarpsN : warp % D::kWarpsN;
    static_assert(!PRODUCT || (D::kThreads == 256 && (D::kWarpsN == 4 || D::kWarpsN == 8)), "the mapping above");
    const int g = lane >> 2, t = lane & 3;

    double acc[D::kMi][D::kNi][2];
#pragma unroll
    for (int mi = 0; mi < D::kMi; ++mi)
#pragma unroll
        for (int ni = 0; ni < D::kNi; ++ni) {
            if (PRODUCT) {
                acc[mi][ni][0] = acc[mi][ni][1] = 0.0;
            } else {
                const int r = wm * WM + mi * 8 + g;
                const int c = wn * WN + ni * 8 + 2 * t;
                const double2 v = *reinterpret_cast<const double2*>(C + (size_t)r * ldc + c);
                acc[mi][ni][0] = -v.x;
                acc[mi][ni][1] = -v.y;
            }
        }

    const int ktiles = K / BK;
    // PRODUCT 1: columns wn*WN .. wn*WN+WN-1 of B vanish past row wn*WN+WN-1; 2: before row wn*WN
    const int kt_warp = PRODUCT == 1 ? min(ktiles, (wn * WN + WN + BK - 1) / BK) : ktiles;
    const int kt_first = PRODUCT == 2 ? wn * WN / BK : 0;
    auto load_stage = [&](int stage, int kt) {
        const int kc = kt * BK;
#pragma unroll
        for (int q = 0; q < D::kChunks / D::kThreads; ++q) {
            const int e = tid + D::kThreads * q;
            const int row = e >> 3, ch = e & 7;
            if (row < TM) {
                cp_async16(As + (stage * TM + row) * SPAD + ch * 2, Ag + (size_t)row * lda + kc + ch * 2);
            } else if (PRODUCT == 1) {
                const int eb = e - TM * (BK / 2), kr = eb / (TN / 2), cc = 2 * (eb % (TN / 2));
                cp_async16(Bs + stage * D::kBStage + kr * D::kBRow + cc, Bg + (size_t)(kc + kr) * ldb + cc);
            } else {
                cp_async16(Bs + stage * D::kBStage + (row - TM) * SPAD + ch * 2,
                           Bg + (size_t)(row - TM) * ldb + kc + ch * 2);
            }
        }
    };
#pragma unroll
    for (int s = 0; s < ST - 1; ++s) {
        if (s < ktiles) load_stage(s, s);
        cp_async_commit();
    }
    for (int kt = 0; kt < ktiles; ++kt) {
        cp_async_wait<ST - 2>();
        __syncthreads();
        {
            const int nk = kt + ST - 1;
            if (nk < ktiles) load_stage(nk % ST, nk);
            cp_async_commit();
        }
        if (kt >= kt_first && kt < kt_warp) {
            const double* as = As + (kt % ST) * TM * SPAD + (wm * WM + g) * SPAD + t;
            const double* bs = Bs + (kt % ST) * D::kBStage +
                               (PRODUCT == 1 ? t * D::kBRow + wn * WN + g : (wn * WN + g) * SPAD + t);
#pragma unroll
            for (int kk = 0; kk < BK / 4; ++kk) {
                double a[D::kMi], b[D::kNi];
#pragma unroll
                for (int mi = 0; mi < D::kMi; ++mi) a[mi] = as[mi * 8 * SPAD + kk * 4];
#pragma unroll
                for (int ni = 0; ni < D::kNi; ++ni) b[ni] = PRODUCT == 1 ? bs[kk * 4 * D::kBRow + ni * 8] : bs[ni * 8 * SPAD + kk * 4];
#pragma unroll
                for (int mi = 0; mi < D::kMi; ++mi)
#pragma unroll
                    for (int ni = 0; ni < D::kNi; ++ni) dmma884(acc[mi][ni], a[mi], b[ni]);
            }
        }
    }
    cp_async_wait<0>();
    __syncthreads();  // every load of A has landed before C (possibly A) is written
#pragma unroll
    for (int mi = 0; mi < D::kMi; ++mi)
#pragma unroll
        for (int ni = 0; ni < D::kNi; ++ni) {
            const int r = wm * WM + mi * 8 + g;
            const int c = wn * WN + ni * 8 + 2 * t;
            const double v0 = PRODUCT ? acc[mi][ni][0] : -acc[mi][ni][0];
            const double v1 = PRODUCT ? acc[mi][ni][1] : -acc[mi][ni][1];
            double* p = C + (size_t)r * ldc + c;
            if (!lower || c + 1 + shift <= r) {
                *reinterpret_cast<double2*>(p) = make_double2(v0, v1);
            } else if (c + shift <= r) {
                p[0] = v0;
            }
        }
}

// Trailing update, two CTAs an SM: 128 x 64 tiles, 8 warps of 32 x 32, 3 stages.
// Each CTA's C preload and store overlap the other CTA's tensor work.
constexpr int kUTM = 128, kUTN = 64, kUWM = 32, kUWN = 32, kUST = 3;
using UTile = DTile<kUTM, kUTN, kUWM, kUWN, kUST>;
// An update too small to give every SM a tile is on the factor's critical path and takes
// one tile's time: 32 x 32 tiles of four warps then (a column of 20 blocks of 128: 15 -> 5
// us).  Above that the larger tiles' reuse wins.
using USmall = DTile<32, 32, 16, 16, 3>;

// Work list of a trailing update.  Column mode (the factor driver): the pairs
// (r, c) of the columns c in [colStart, colEnd), c <= r < nb, column by column.
// Row mode (the operator entry points, MatrixMatrixOperations.cpp:146-906): GEMM
// pairs (r, c), r in [gemmStart, gemmStart+gemmCount), blockRow < c < r, then
// SYRK diagonal blocks j in [syrkStart, syrkStart+syrkCount).
struct UpdateArgs {
    double* A;
    int64_t blockID;  // diagonal block of column blockRow (the panel's column)
    int blockRow, nb, bsz;
    int rowMode;
    int colStart, colEnd;            // column mode
    int64_t gemmPairs, pairBase;     // row mode
    int syrkStart;
    int tilesM, tilesN;
    int64_t totalPairs;
};

__device__ __forceinline__ void decode_pair(const UpdateArgs& a, int64_t pair, int* r, int* c) {
    if (a.rowMode) {
        if (pair < a.gemmPairs) {
            const int64_t tt = pair + a.pairBase;
            const int u = tri_root(tt);
            *r = a.blockRow + 1 + (u + 1);
            *c = a.blockRow + 1 + (int)(tt - (int64_t)u * (u + 1) / 2);
        } else {
            *r = *c = a.syrkStart + (int)(pair - a.gemmPairs);
        }
        return;
    }
    // column c holds nb - c pairs: the largest c with offset(c) <= pair
    auto offset = [&](int cc) -> int64_t {
        return (int64_t)(cc - a.colStart) * a.nb - ((int64_t)cc * (cc - 1) - (int64_t)a.colStart * (a.colStart - 1)) / 2;
    };
    int lo = a.colStart, hi = a.colEnd - 1;
    while (lo < hi) {
        const int mid = (lo + hi + 1) >> 1;
        if (offset(mid) <= pair) lo = mid; else hi = mid - 1;
    }
    *c = lo;
    *r = lo + (int)(pair - offset(lo));
}

template <int TM, int TN, int WM, int WN, int ST, int CTAS>
__global__ void __launch_bounds__(DTile<TM, TN, WM, WN, ST>::kThreads, CTAS) update_dmma_kernel(UpdateArgs a) {
    extern __shared__ __align__(16) double smem[];
    const int tpb = a.tilesM * a.tilesN;
    const int64_t pair = blockIdx.x / tpb;
    const int tile = (int)(blockIdx.x % tpb);
    int r, c;
    decode_pair(a, pair, &r, &c);
    const int ti = tile / a.tilesN, tj = tile % a.tilesN;
    const int shift = tj * TN - ti * TM;  // tile column offset minus row offset inside the block
    const bool diag = r == c;
    if (diag && shift > TM - 1) return;      // entirely above the diagonal
    const bool lower = diag && shift + TN - 1 > 0;
    const size_t bb = (size_t)a.bsz * a.bsz;
    double* C = a.A + (size_t)block_id(r, c, a.nb) * bb + (size_t)ti * TM * a.bsz + (size_t)tj * TN;
    const double* Ag = a.A + (size_t)(a.blockID + (r - a.blockRow)) * bb + (size_t)ti * TM * a.bsz;
    const double* Bg = a.A + (size_t)(a.blockID + (c - a.blockRow)) * bb + (size_t)tj * TN * a.bsz;
    dmma_tile_t<TM, TN, WM, WN, ST, 0>(C, a.bsz, Ag, a.bsz, Bg, a.bsz, a.bsz, lower, shift, smem);
}
constexpr auto update_large = update_dmma_kernel<kUTM, kUTN, kUWM, kUWN, kUST, 2>;
constexpr auto update_small = update_dmma_kernel<32, 32, 16, 16, 3, 4>;

// Panel TRSM as a tensor-core product: B <- B Y with Y = L_kk^-T (row major, upper
// triangular), in place; one CTA per ROWS rows of a panel block: 64, or 32 where 64 leave
// SMs without work.
template <int BSZ, int ROWS>
using TrsmTile = DTile<ROWS, BSZ, 32, ROWS * BSZ / 256, 3>;

template <int BSZ, int ROWS>
__global__ void __launch_bounds__(256, 1) trsm_dmma_kernel(double* A, int64_t firstBlock, const double* __restrict__ Y,
                                                           double* Lkk) {
    extern __shared__ __align__(16) double smem[];
    if (Lkk) {
        // the zeros above the 32 x 32 diagonal blocks of L_kk, off the chain that produced it
        constexpr int kT = BSZ / 32, kPairs = kT * (kT - 1) / 2;
        for (int u = blockIdx.x; u < kPairs; u += gridDim.x) {
            const int c = tri_root(u) + 1, r = u - c * (c - 1) / 2;  // r < c
            for (int e = threadIdx.x; e < 512; e += 256)
                *reinterpret_cast<double2*>(Lkk + (size_t)(32 * r + e / 16) * BSZ + 32 * c + 2 * (e % 16)) =
                    make_double2(0.0, 0.0);
        }
    }
    constexpr int kSlabs = BSZ / ROWS;
    const int64_t item = blockIdx.x / kSlabs;
    const int slab = blockIdx.x % kSlabs;
    double* B = A + (size_t)(firstBlock + item) * BSZ * BSZ + (size_t)slab * ROWS * BSZ;
    dmma_tile_t<ROWS, BSZ, 32, ROWS * BSZ / 256, 3, 1>(B, BSZ, B, BSZ, Y, BSZ, BSZ, false, 0, smem);
}

// L_rk <- L_rk Y_k^T for every off-diagonal block, one CTA per 64 rows of a block
template <int BSZ>
__global__ void __launch_bounds__(256, 1) scale_panels_kernel(double* L, int nb, const double* __restrict__ Y) {
    extern __shared__ __align__(16) double smem[];
    constexpr int kRows = 64, kSlabs = BSZ / kRows;
    const int64_t pair = blockIdx.x / kSlabs;  // (r, k), r > k: triangle of nb - 1 columns
    int i, k;
    block_coords(pair, nb - 1, &i, &k);
    double* B = L + ((size_t)block_id(i + 1, k, nb) * BSZ + (size_t)(blockIdx.x % kSlabs) * kRows) * BSZ;
    dmma_tile_t<kRows, BSZ, 32, kRows * BSZ / 256, 3, 2>(B, BSZ, B, BSZ, Y + (size_t)k * BSZ * BSZ, BSZ, BSZ, false, 0,
                                                         smem);
}

// scalar fallback (any bsz): one thread per output element; SYRK follows
// MatrixMatrixOperations.cpp:346-355 (value -= c_ik c_jk in k order), GEMM
// follows :893-900 (sum from zero, subtracted once)
__global__ void update_scalar_kernel(UpdateArgs a) {
    const int64_t bb = (int64_t)a.bsz * a.bsz;
    const int64_t pair = blockIdx.y + (int64_t)blockIdx.z * 65535;
    if (pair >= a.totalPairs) return;
    int r, c;
    decode_pair(a, pair, &r, &c);
    const int64_t e = blockIdx.x * (int64_t)blockDim.x + threadIdx.x;
    if (e >= bb) return;
    const int i = (int)(e / a.bsz), j = (int)(e % a.bsz);
    double* C = a.A + block_id(r, c, a.nb) * bb;
    const double* Rk = a.A + (a.blockID + (r - a.blockRow)) * bb;
    const double* Ck = a.A + (a.blockID + (c - a.blockRow)) * bb;
    if (r == c) {
        if (i < j) return;
        double v = C[(size_t)i * a.bsz + j];
        for (int k = 0; k < a.bsz; ++k) v = v - Rk[(size_t)i * a.bsz + k] * Rk[(size_t)j * a.bsz + k];
        C[(size_t)i * a.bsz + j] = v;
    } else {
        double v = 0.0;
        for (int k = 0; k < a.bsz; ++k) v += Rk[(size_t)i * a.bsz + k] * Ck[(size_t)j * a.bsz + k];
        C[(size_t)i * a.bsz + j] -= v;
    }
}

bool attrs_done[64] = {};
hs_status set_attrs() {
    int dev = 0;
    HS_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && attrs_done[dev]) return HS_OK;
    HS_CUDA(cudaFuncSetAttribute(update_large, cudaFuncAttributeMaxDynamicSharedMemorySize, UTile::kSmem));
    HS_CUDA(cudaFuncSetAttribute(update_small, cudaFuncAttributeMaxDynamicSharedMemorySize, USmall::kSmem));
    HS_CUDA(cudaFuncSetAttribute(trsm_dmma_kernel<128, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 TrsmTile<128, 64>::kSmem));
    HS_CUDA(cudaFuncSetAttribute(trsm_dmma_kernel<256, 64>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 TrsmTile<256, 64>::kSmem));
    HS_CUDA(cudaFuncSetAttribute(trsm_dmma_kernel<128, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 TrsmTile<128, 32>::kSmem));
    HS_CUDA(cudaFuncSetAttribute(trsm_dmma_kernel<256, 32>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 TrsmTile<256, 32>::kSmem));
    HS_CUDA(cudaFuncSetAttribute(scale_panels_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 TrsmTile<128, 64>::kSmem));
    HS_CUDA(cudaFuncSetAttribute(scale_panels_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 TrsmTile<256, 64>::kSmem));
    HS_CUDA(cudaFuncSetAttribute(trsm_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)trsm_smem(256)));
    HS_CUDA(cudaFuncSetAttribute(potrf_smem_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize,
                                 (int)(128 * 129 * sizeof(double))));
    if (dev >= 0 && dev < 64) attrs_done[dev] = true;
    return HS_OK;
}

hs_status launch_trsm_args(hs_ctx ctx, const TrsmArgs& ta, int items, cudaStream_t s) {
    ctx->launches += 1;
    HS_REQUIRE(ta.n <= 256, "TRSM supports triangles up to 256");
    const size_t smem = trsm_smem(ta.n);
    trsm_kernel<<<items * ta.slabs, 256, smem, s>>>(ta);
    HS_CHECK_LAUNCH("trsm");
    return HS_OK;
}

hs_status potrf_small(hs_ctx ctx, double* blk, int ld, int n, int valid, long long row_base, cudaStream_t s) {
    const size_t smem = (size_t)n * (n + 1) * sizeof(double);
    ctx->launches += 1;
    potrf_smem_kernel<<<1, 512, smem, s>>>(blk, ld, n, valid, ctx->d_info, row_base);
    HS_CHECK_LAUNCH("potrf");
    return HS_OK;
}

}  // namespace

static hs_status potrf_impl(hs_ctx ctx, double* A, int blockID, int blockRow, cudaStream_t s) {
    hs_status st = set_attrs();
    if (st != HS_OK) return st;
    const int bsz = ctx->bsz;
    double* blk = A + (size_t)blockID * bsz * bsz;
    const long long row_base = (long long)blockRow * bsz;
    const int64_t rem = ctx->N - row_base;
    const int valid = rem <= 0 ? 0 : (rem < bsz ? (int)rem : bsz);
    // The on-chip block reads and writes 16 bytes at a time; a matrix that is aligned to its
    // entries only takes the kernels of the other block sizes.
    if ((bsz == 128 || bsz == 256) && reinterpret_cast<uintptr_t>(blk) % 16 == 0) {
        DiagFactor f;
        f.in64 = f.L = blk;
        f.in_place = 1;
        f.row_base = row_base;
        return launch_diag_factor(ctx, f, s);
    }
    if (bsz <= 128) return potrf_small(ctx, blk, bsz, bsz, valid, row_base, s);
    ctx->launches += 1;
    potrf_global_kernel<<<1, 1024, 0, s>>>(blk, bsz, valid, ctx->d_info, row_base);
    HS_CHECK_LAUNCH("potrf");
    return HS_OK;
}

hs_status launch_potrf(hs_ctx ctx, double* A, int blockID, int blockRow, cudaStream_t s) {
    const double n = ctx->bsz;
    prof_begin(ctx, s, HS_KERNEL_POTRF);
    hs_status st = potrf_impl(ctx, A, blockID, blockRow, s);
    prof_end(ctx, s, HS_KERNEL_POTRF, n * n * n / 3.0, 2.0 * n * n * 8.0);
    return st;
}

hs_status launch_trsm_dmma(hs_ctx ctx, double* A, int64_t firstBlock, int blockCount, const double* Y, double* Lkk,
                           cudaStream_t s) {
    if (blockCount <= 0) return HS_OK;
    hs_status st = set_attrs();
    if (st != HS_OK) return st;
    const int bsz = ctx->bsz;
    HS_REQUIRE(bsz == 128 || bsz == 256, "the tensor-core TRSM needs matrixBlockSize 128 or 256");
    const double n = bsz;
    prof_begin(ctx, s, HS_KERNEL_TRSM);
    ctx->launches += 1;
    const int64_t wide = (int64_t)blockCount * (bsz / 64);
    if (wide <= ctx->num_sms) {
        const unsigned grid = (unsigned)(2 * wide);
        if (bsz == 256)
            trsm_dmma_kernel<256, 32><<<grid, 256, TrsmTile<256, 32>::kSmem, s>>>(A, firstBlock, Y, Lkk);
        else
            trsm_dmma_kernel<128, 32><<<grid, 256, TrsmTile<128, 32>::kSmem, s>>>(A, firstBlock, Y, Lkk);
    } else if (bsz == 256) {
        trsm_dmma_kernel<256, 64><<<(unsigned)wide, 256, TrsmTile<256, 64>::kSmem, s>>>(A, firstBlock, Y, Lkk);
    } else {
        trsm_dmma_kernel<128, 64><<<(unsigned)wide, 256, TrsmTile<128, 64>::kSmem, s>>>(A, firstBlock, Y, Lkk);
    }
    HS_CHECK_LAUNCH("trsm_dmma");
    // algorithmic work: the triangular solve's n^3 flops a block
    prof_end(ctx, s, HS_KERNEL_TRSM, blockCount * n * n * n, (2.0 * blockCount + 1.0) * n * n * 8.0);
    return HS_OK;
}

hs_status launch_scale_panels(hs_ctx ctx, double* L, const double* Y, cudaStream_t s) {
    const int nb = ctx->nb, bsz = ctx->bsz;
    if (nb < 2) return HS_OK;
    hs_status st = set_attrs();
    if (st != HS_OK) return st;
    HS_REQUIRE(bsz == 128 || bsz == 256, "the tensor-core panels need matrixBlockSize 128 or 256");
    const int64_t blocks = total_blocks(nb - 1), grid = blocks * (bsz / 64);
    HS_REQUIRE(grid < (1LL << 31), "too many blocks");
    const double n = bsz;
    prof_begin(ctx, s, HS_KERNEL_ADJOINT);
    ctx->launches += 1;
    if (bsz == 256)
        scale_panels_kernel<256><<<(unsigned)grid, 256, TrsmTile<256, 64>::kSmem, s>>>(L, nb, Y);
    else
        scale_panels_kernel<128><<<(unsigned)grid, 256, TrsmTile<128, 64>::kSmem, s>>>(L, nb, Y);
    HS_CHECK_LAUNCH("scale_panels");
    prof_end(ctx, s, HS_KERNEL_ADJOINT, blocks * n * n * n, 2.0 * blocks * n * n * 8.0);
    return HS_OK;
}

hs_status launch_trsm(hs_ctx ctx, double* A, int blockID, int blockRow, int blockStart, int blockCount,
                      cudaStream_t s) {
    if (blockCount <= 0) return HS_OK;
    hs_status st = set_attrs();
    if (st != HS_OK) return st;
    const int bsz = ctx->bsz;
    HS_REQUIRE(bsz <= 256, "TRSM supports matrixBlockSize up to 256");
    const size_t bb = (size_t)bsz * bsz;
    if (bsz == 128 || bsz == 256) {
        // on the FP64 tensor pipe: Y = L_kk^-T once, then B <- B Y block by block
        st = ensure_scratch(ctx, kSmallScratch + kDiagScratchBlocks * bb * sizeof(double));
        if (st != HS_OK) return st;
        double* Y = reinterpret_cast<double*>(static_cast<char*>(ctx->scratch) + kSmallScratch);
        st = launch_diag_inverse(ctx, A + (size_t)blockID * bb, Y, Y + bb, s);
        if (st != HS_OK) return st;
        return launch_trsm_dmma(ctx, A, (int64_t)blockID + (blockStart - blockRow), blockCount, Y, nullptr, s);
    }
    TrsmArgs ta{A + (size_t)blockID * bb, bsz, bsz, A, bsz, (int64_t)blockID + (blockStart - blockRow),
                (bsz + kTrsmRows - 1) / kTrsmRows, bsz, (int64_t)bb};
    const double n = bsz;
    prof_begin(ctx, s, HS_KERNEL_TRSM);
    st = launch_trsm_args(ctx, ta, blockCount, s);
    prof_end(ctx, s, HS_KERNEL_TRSM, blockCount * n * n * n, (2.0 * blockCount + 1.0) * n * n * 8.0);
    return st;
}

namespace {

// launches the update of `a` (totalPairs set) with its algorithmic flops / bytes
hs_status run_update(hs_ctx ctx, UpdateArgs& a, double flops, double bytes, cudaStream_t s) {
    if (a.totalPairs <= 0) return HS_OK;
    const bool dmma = ctx->bsz % kUTM == 0;
    a.tilesM = dmma ? ctx->bsz / kUTM : 1;
    a.tilesN = dmma ? ctx->bsz / kUTN : 1;
    const bool small = dmma && a.totalPairs * a.tilesM * a.tilesN <= ctx->num_sms;
    if (small) a.tilesM = a.tilesN = ctx->bsz / 32;
    const int64_t grid = a.totalPairs * a.tilesM * a.tilesN;
    HS_REQUIRE(grid < (1LL << 31), "trailing update too large for one launch");
    prof_begin(ctx, s, HS_KERNEL_UPDATE);
    ctx->launches += 1;
    if (dmma) {
        if (small)
            update_small<<<(unsigned)grid, USmall::kThreads, USmall::kSmem, s>>>(a);
        else
            update_large<<<(unsigned)grid, UTile::kThreads, UTile::kSmem, s>>>(a);
        HS_CHECK_LAUNCH("update_dmma");
    } else {
        const int64_t bb = (int64_t)ctx->bsz * ctx->bsz;
        const int64_t total = a.totalPairs;
        dim3 g((unsigned)((bb + 255) / 256), (unsigned)(total < 65535 ? total : 65535),
               (unsigned)((total + 65534) / 65535));
        update_scalar_kernel<<<g, 256, 0, s>>>(a);
        HS_CHECK_LAUNCH("update_scalar");
    }
    prof_end(ctx, s, HS_KERNEL_UPDATE, flops, bytes);
    return HS_OK;
}

}  // namespace

hs_status launch_update(hs_ctx ctx, double* A, int blockID, int blockRow, int syrkStart, int syrkCount,
                        int gemmStart, int gemmCount, cudaStream_t s) {
    hs_status st = set_attrs();
    if (st != HS_OK) return st;
    UpdateArgs a{};
    a.A = A;
    a.blockID = blockID;
    a.blockRow = blockRow;
    a.nb = ctx->nb;
    a.bsz = ctx->bsz;
    a.rowMode = 1;
    int64_t pairs = 0;
    if (gemmCount > 0) {
        // rows r' = r - blockRow - 1 in [g0, g0 + gemmCount) own r' pairs each
        const int64_t g0 = gemmStart - blockRow - 1;
        const int64_t g1 = g0 + gemmCount;
        a.pairBase = g0 * (g0 - 1) / 2;
        pairs = g1 * (g1 - 1) / 2 - a.pairBase;
    }
    a.gemmPairs = pairs;
    a.syrkStart = syrkStart;
    const int64_t syrkN = syrkCount > 0 ? syrkCount : 0;
    a.totalPairs = pairs + syrkN;
    // algorithmic work: 2 bsz^3 per GEMM pair, bsz^2 (bsz + 1) per SYRK block;
    // bytes: read + write of every output block plus the panel column once
    const double n = ctx->bsz;
    const double flops = (double)pairs * 2.0 * n * n * n + (double)syrkN * n * n * (n + 1.0);
    const int64_t panel = (gemmCount > 0 ? gemmCount + 1 : 0) > syrkN ? (gemmCount + 1) : syrkN;
    const double bytes = ((double)pairs * 2.0 + (double)syrkN * 2.0 + (double)panel) * n * n * 8.0;
    return run_update(ctx, a, flops, bytes, s);
}

hs_status launch_update_cols(hs_ctx ctx, double* A, int blockID, int blockRow, int colStart, int colEnd,
                             cudaStream_t s) {
    hs_status st = set_attrs();
    if (st != HS_OK) return st;
    const int nb = ctx->nb;
    HS_REQUIRE(blockRow < colStart && colStart <= colEnd && colEnd <= nb, "columns outside the trailing matrix");
    UpdateArgs a{};
    a.A = A;
    a.blockID = blockID;
    a.blockRow = blockRow;
    a.nb = nb;
    a.bsz = ctx->bsz;
    a.rowMode = 0;
    a.colStart = colStart;
    a.colEnd = colEnd;
    int64_t pairs = 0;
    for (int c = colStart; c < colEnd; ++c) pairs += nb - c;
    a.totalPairs = pairs;
    const double n = ctx->bsz;
    const int64_t syrkN = colEnd - colStart;
    const double flops = (double)(pairs - syrkN) * 2.0 * n * n * n + (double)syrkN * n * n * (n + 1.0);
    const double bytes = ((double)pairs * 2.0 + (double)(nb - colStart)) * n * n * 8.0;
    return run_update(ctx, a, flops, bytes, s);
}

}  // namespace hs
