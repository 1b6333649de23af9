// k_predict.cu — GP prediction: the test kernel matrix K*, the dense
// matrix-vector product of the prediction, and a fused predictive mean that
// never stores K*.
//
// Replaces MatrixGenerator::generateTestKernelMatrix
// (src/utility/MatrixGenerator.cpp:163-213: K*[j*N + i] = sf2 exp(-0.5/l^2 *
// sum_k (x_ik - x*_jk)^2), k ascending, no noise term) and
// MatrixVectorOperations::matrixVectorGP (src/kernel/MatrixVectorOperations.cpp:
// 379-395: result[i] = sum_k A[i*n + k] b[k] for i < m), the two steps of
// GaussianProcess::start's prediction (src/gaussianProcess/GaussianProcess.cpp:
// 42-54).  The inputs are row-major X (N x d) and X* (N_test x d); the
// reference's 8-sample sliding window is one instance, ARD lengthscales the
// generalisation (each difference scaled by 1/l_k, then exp(-0.5 * distance)).
#include <algorithm>
#include <type_traits>

#include "hs_internal.cuh"

namespace hs {
namespace {

constexpr int kMaxD = 64;
constexpr int kPredThreads = 256;

__device__ __forceinline__ double sq_dist(const double* __restrict__ a, const double* __restrict__ bT, int stride,
                                          int d, int ard, const double* __restrict__ w) {
    double dist = 0.0;
    for (int k = 0; k < d; ++k) {
        const double t = ard ? (a[k] - bT[(size_t)k * stride]) * w[k] : a[k] - bT[(size_t)k * stride];
        dist += t * t;
    }
    return dist;
}

// K*: CTA = 16 test rows x 256 training columns; X* rows and the X columns
// (transposed) staged in shared memory; each warp writes 256 contiguous bytes
// of one K* row per instruction.
__global__ void __launch_bounds__(kPredThreads) test_kernel_matrix_kernel(
    const double* __restrict__ X, int64_t N, const double* __restrict__ Xt, int64_t Nt, int d, int ard,
    const double* __restrict__ w, double scale, double sf2, double* __restrict__ Ks) {
    extern __shared__ double sm[];
    constexpr int TJ = 16, TI = 256;
    double* xt = sm;                    // [TJ][d]
    double* xT = sm + TJ * d;           // [d][TI]
    __shared__ double ws[kMaxD];
    const int64_t j0 = (int64_t)blockIdx.y * TJ, i0 = (int64_t)blockIdx.x * TI;
    for (int e = threadIdx.x; e < TJ * d; e += blockDim.x) {
        const int r = e / d, k = e % d;
        xt[e] = (j0 + r < Nt) ? Xt[(j0 + r) * d + k] : 0.0;
    }
    for (int e = threadIdx.x; e < TI * d; e += blockDim.x) {
        const int r = e / d, k = e % d;
        xT[(size_t)k * TI + r] = (i0 + r < N) ? X[(i0 + r) * d + k] : 0.0;
    }
    if (threadIdx.x < d) ws[threadIdx.x] = ard ? w[threadIdx.x] : 1.0;
    __syncthreads();
    const int il = threadIdx.x;
    const int64_t i = i0 + il;
    if (i >= N) return;
    for (int jl = 0; jl < TJ; ++jl) {
        const int64_t j = j0 + jl;
        if (j >= Nt) break;
        const double dist = sq_dist(xt + jl * d, xT + il, TI, d, ard, ws);
        __stcs(Ks + j * N + i, sf2 * exp((ard ? -0.5 : scale) * dist));
    }
}

// result[i] = sum_k A[i*n + k] b[k]: one warp per row, lanes stride the row,
// fixed-order butterfly reduction
__global__ void __launch_bounds__(kPredThreads) matvec_rows_kernel(const double* __restrict__ A,
                                                                   const double* __restrict__ b,
                                                                   double* __restrict__ result, int64_t n, int64_t m) {
    const int lane = threadIdx.x & 31;
    const int64_t warps = (int64_t)gridDim.x * (blockDim.x >> 5);
    for (int64_t row = (int64_t)blockIdx.x * (blockDim.x >> 5) + (threadIdx.x >> 5); row < m; row += warps) {
        const double* a = A + row * n;
        double s0 = 0.0, s1 = 0.0, s2 = 0.0, s3 = 0.0;
        int64_t k = lane;
        for (; k + 96 < n; k += 128) {
            s0 = fma(__ldcs(a + k), b[k], s0);
            s1 = fma(__ldcs(a + k + 32), b[k + 32], s1);
            s2 = fma(__ldcs(a + k + 64), b[k + 64], s2);
            s3 = fma(__ldcs(a + k + 96), b[k + 96], s3);
        }
        for (; k < n; k += 32) s0 = fma(__ldcs(a + k), b[k], s0);
        double s = (s0 + s1) + (s2 + s3);
        for (int o = 16; o > 0; o >>= 1) s += __shfl_xor_sync(0xffffffffu, s, o);
        if (lane == 0) result[row] = s;
    }
}

// fused predictive mean: mean[j] = sum_i k(x*_j, x_i) alpha_i without storing K*.  A CTA
// takes 64 test points and one of `splits` ranges of the training points, in steps of 64;
// a thread 4 x 4 pairs, so that each staged value serves four distances (with one pair a
// thread the kernel was bound by shared memory, at an eighth of the FP64 pipe's rate).  The
// ranges' parts go to part[split][j] and are summed in order by sum_splits_kernel.
// N=16384, 5000 test points, d=16: 2000 -> 388 us (FP64 pipe alone: ~260 us).
constexpr int kPredTile = 64;
__global__ void __launch_bounds__(kPredThreads, 2) predict_mean_kernel(
    const double* __restrict__ X, int64_t N, const double* __restrict__ Xt, int64_t Nt, int d, int ard,
    const double* __restrict__ w, double scale, double sf2, const double* __restrict__ alpha, int64_t range,
    double* __restrict__ part) {
    extern __shared__ __align__(16) double sm[];
    constexpr int T = kPredTile;
    double* xt = sm;            // [d][T] test points, transposed
    double* xi = xt + d * T;    // [2][d][T] training points, transposed
    __shared__ double al[2][T], ws[kMaxD];
    const int tid = threadIdx.x, tx = tid & 15, ty = tid >> 4;
    const int64_t j0 = (int64_t)blockIdx.x * T;
    const int64_t i_begin = (int64_t)blockIdx.y * range, i_end = min(N, i_begin + range);
    // neighbouring threads take neighbouring points of one feature: no bank conflicts
    auto stage = [&](double* dst, const double* src, int64_t first, int64_t count) {
        for (int e = tid; e < T * d; e += kPredThreads) {
            const int r = e % T, k = e / T;
            dst[e] = first + r < count ? src[(first + r) * d + k] : 0.0;
        }
    };
    stage(xt, Xt, j0, Nt);
    if (tid < d) ws[tid] = ard ? w[tid] : 1.0;
    double acc[4] = {0.0, 0.0, 0.0, 0.0};
    int buf = 0;
    for (int64_t i0 = i_begin; i0 < i_end; i0 += T, buf ^= 1) {
        double* xb = xi + buf * d * T;
        stage(xb, X, i0, i_end);
        if (tid < T) al[buf][tid] = i0 + tid < i_end ? alpha[i0 + tid] : 0.0;
        __syncthreads();  // (the other buffer is free: every thread has passed its use)
        double dist[4][4];
#pragma unroll
        for (int p = 0; p < 4; ++p)
#pragma unroll
            for (int q = 0; q < 4; ++q) dist[p][q] = 0.0;
        auto features = [&](auto with_weight) {
#pragma unroll 2
            for (int k = 0; k < d; ++k) {
                const double2 t0 = *reinterpret_cast<const double2*>(xt + k * T + 4 * ty);
                const double2 t1 = *reinterpret_cast<const double2*>(xt + k * T + 4 * ty + 2);
                const double2 u0 = *reinterpret_cast<const double2*>(xb + k * T + 2 * tx);
                const double2 u1 = *reinterpret_cast<const double2*>(xb + k * T + 32 + 2 * tx);
                const double tv[4] = {t0.x, t0.y, t1.x, t1.y}, uv[4] = {u0.x, u0.y, u1.x, u1.y};
                const double wk = decltype(with_weight)::value ? ws[k] : 1.0;
#pragma unroll
                for (int p = 0; p < 4; ++p)
#pragma unroll
                    for (int q = 0; q < 4; ++q) {
                        double t = tv[p] - uv[q];
                        if (decltype(with_weight)::value) t *= wk;
                        dist[p][q] = fma(t, t, dist[p][q]);
                    }
            }
        };
        if (ard)
            features(std::true_type{});
        else
            features(std::false_type{});
        const double sc = ard ? -0.5 : scale;
#pragma unroll
        for (int q = 0; q < 4; ++q) {
            const int il = (q >> 1) * 32 + 2 * tx + (q & 1);
            const double a = al[buf][il];
            if (i0 + il < i_end) {
#pragma unroll
                for (int p = 0; p < 4; ++p) acc[p] = fma(sf2 * exp(sc * dist[p][q]), a, acc[p]);
            }
        }
    }
    // over the 16 threads of a row of the tile, in a tree
#pragma unroll
    for (int p = 0; p < 4; ++p) {
        for (int o = 8; o > 0; o >>= 1) acc[p] += __shfl_xor_sync(0xffffffffu, acc[p], o);
        if (tx == 0 && j0 + 4 * ty + p < Nt) part[(int64_t)blockIdx.y * Nt + j0 + 4 * ty + p] = acc[p];
    }
}

__global__ void sum_splits_kernel(const double* __restrict__ part, int64_t Nt, int splits, double* __restrict__ mean) {
    for (int64_t j = blockIdx.x * (int64_t)blockDim.x + threadIdx.x; j < Nt; j += (int64_t)gridDim.x * blockDim.x) {
        double s = 0.0;
        for (int q = 0; q < splits; ++q) s += part[(int64_t)q * Nt + j];
        mean[j] = s;
    }
}

struct Scales {
    int ard = 0;
    double scale = 0.0;
    double* w = nullptr;  // device, d
};

hs_status make_scales(hs_ctx ctx, int d, const double* ell, int n_ell, Scales* out) {
    HS_REQUIRE(d >= 1 && d <= kMaxD, "d must be in [1, 64]");
    HS_REQUIRE(n_ell == 1 || n_ell == d, "n_ell must be 1 or d");
    for (int k = 0; k < n_ell; ++k) HS_REQUIRE(ell[k] > 0.0, "lengthscales must be positive");
    out->ard = (n_ell == d && d > 1) ? 1 : 0;
    out->scale = -0.5 / (ell[0] * ell[0]);
    hs_status st = ensure_scratch(ctx, kSmallScratch);
    if (st != HS_OK) return st;
    double* w = reinterpret_cast<double*>(static_cast<char*>(ctx->scratch) + kConstOffset);
    if (out->ard) {
        double hw[kMaxD];
        for (int k = 0; k < d; ++k) hw[k] = 1.0 / ell[k];
        HS_CUDA(cudaMemcpyAsync(w, hw, d * sizeof(double), cudaMemcpyHostToDevice, ctx->stream));
        HS_CUDA(cudaStreamSynchronize(ctx->stream));  // hw is a stack buffer
    }
    out->w = w;
    return HS_OK;
}

}  // namespace
}  // namespace hs

using namespace hs;

extern "C" {

hs_status hs_gp_test_kernel_matrix(hs_ctx ctx, const double* X, const double* X_test, int64_t N_test, int d,
                                   const double* ell, int n_ell, double sf2, double* K_star) {
    hs_status st = require_ctx(ctx, "hs_gp_test_kernel_matrix");
    if (st != HS_OK) return st;
    if (!X || !X_test || !ell || !K_star || N_test < 0) {
        set_error("hs_gp_test_kernel_matrix: null pointer or negative N_test");
        return HS_ERR_INVALID_ARG;
    }
    if (N_test == 0) return HS_OK;
    Scales sc;
    if ((st = make_scales(ctx, d, ell, n_ell, &sc)) != HS_OK) return st;
    const int64_t N = ctx->N;
    dim3 grid((unsigned)((N + 255) / 256), (unsigned)((N_test + 15) / 16));
    HS_REQUIRE(grid.y <= 65535, "N_test too large (at most 1048560)");
    const size_t smem = (size_t)(16 + 256) * d * sizeof(double);
    HS_CUDA(cudaFuncSetAttribute(test_kernel_matrix_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    prof_begin(ctx, ctx->stream, HS_KERNEL_ASSEMBLE);
    ctx->launches += 1;
    test_kernel_matrix_kernel<<<grid, kPredThreads, smem, ctx->stream>>>(X, N, X_test, N_test, d, sc.ard, sc.w,
                                                                        sc.scale, sf2, K_star);
    HS_CHECK_LAUNCH("test_kernel_matrix");
    prof_end(ctx, ctx->stream, HS_KERNEL_ASSEMBLE, (double)N * N_test * (3.0 * d + 20.0),
             (double)N * N_test * 8.0);
    return HS_OK;
}

hs_status hs_matrix_vector_gp(hs_ctx ctx, const double* A, const double* b, double* result, int64_t n, int64_t m) {
    hs_status st = require_ctx(ctx, "hs_matrix_vector_gp");
    if (st != HS_OK) return st;
    if (!A || !b || !result || n < 0 || m < 0) {
        set_error("hs_matrix_vector_gp: null pointer or negative size");
        return HS_ERR_INVALID_ARG;
    }
    if (m == 0) return HS_OK;
    const int64_t rows_per_cta = kPredThreads / 32;
    int64_t grid = (m + rows_per_cta - 1) / rows_per_cta;
    if (grid > 16LL * ctx->num_sms) grid = 16LL * ctx->num_sms;
    prof_begin(ctx, ctx->stream, HS_KERNEL_VECTOR);
    ctx->launches += 1;
    matvec_rows_kernel<<<(unsigned)grid, kPredThreads, 0, ctx->stream>>>(A, b, result, n, m);
    HS_CHECK_LAUNCH("matrix_vector_gp");
    prof_end(ctx, ctx->stream, HS_KERNEL_VECTOR, 2.0 * n * m, 8.0 * ((double)n * m + n + m));
    return HS_OK;
}

hs_status hs_gp_predict(hs_ctx ctx, const double* X, const double* X_test, int64_t N_test, int d, const double* ell,
                        int n_ell, double sf2, const double* alpha, double* mean) {
    hs_status st = require_ctx(ctx, "hs_gp_predict");
    if (st != HS_OK) return st;
    if (!X || !X_test || !ell || !alpha || !mean || N_test < 0) {
        set_error("hs_gp_predict: null pointer or negative N_test");
        return HS_ERR_INVALID_ARG;
    }
    if (N_test == 0) return HS_OK;
    const int64_t N = ctx->N, tiles = (N_test + kPredTile - 1) / kPredTile, steps = (N + kPredTile - 1) / kPredTile;
    HS_REQUIRE(tiles < (1LL << 31), "N_test too large");
    // enough ranges of training points for just under six waves of two CTAs an SM (a wave
    // that is partly empty then costs little), each of at least two steps.  Their parts fit
    // the scratch that a context has anyway: growing it costs a first call more than the
    // last few ranges give (N=16384, 5000 test points: 22 -> 21 ranges)
    const int64_t room = (int64_t)((kScratchSmall - kSmallScratch) / sizeof(double)) / N_test;
    int64_t splits = std::max<int64_t>(1, std::min<int64_t>({12LL * ctx->num_sms / tiles, steps / 2, 512, room}));
    const int64_t range = (steps + splits - 1) / splits * kPredTile;
    splits = (N + range - 1) / range;
    st = ensure_scratch(ctx, kSmallScratch + (splits > 1 ? (size_t)splits * N_test * sizeof(double) : 0));
    if (st != HS_OK) return st;
    double* part = splits > 1 ? reinterpret_cast<double*>(static_cast<char*>(ctx->scratch) + kSmallScratch) : mean;
    // (after the scratch has its size: the weights live in it)
    Scales sc;
    if ((st = make_scales(ctx, d, ell, n_ell, &sc)) != HS_OK) return st;
    const size_t smem = (size_t)3 * kPredTile * d * sizeof(double);
    HS_CUDA(cudaFuncSetAttribute(predict_mean_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)smem));
    prof_begin(ctx, ctx->stream, HS_KERNEL_VECTOR);
    ctx->launches += splits > 1 ? 2 : 1;
    predict_mean_kernel<<<dim3((unsigned)tiles, (unsigned)splits), kPredThreads, smem, ctx->stream>>>(
        X, N, X_test, N_test, d, sc.ard, sc.w, sc.scale, sf2, alpha, range, part);
    if (splits > 1)
        sum_splits_kernel<<<(unsigned)std::min<int64_t>((N_test + 255) / 256, 4LL * ctx->num_sms), 256, 0, ctx->stream>>>(
            part, N_test, (int)splits, mean);
    HS_CHECK_LAUNCH("predict_mean");
    prof_end(ctx, ctx->stream, HS_KERNEL_VECTOR, (double)N * N_test * (3.0 * d + 22.0),
             8.0 * ((double)N * (d + 1) * (double)tiles + N_test * (d + 1.0)));
    return HS_OK;
}

}  // extern "C"
