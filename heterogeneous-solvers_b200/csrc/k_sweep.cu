// k_sweep.cu — a whole forward (out = L^-1 in) or backward (out = L^-T in) substitution
// with a packed FP64 or FP32 factor in one launch, FP64 arithmetic throughout.
//
// Reference path replaced: TriangularSystemSolver.cpp:15-105 (and the preconditioner of the
// mixed-precision form, which has no counterpart there).
//
// With the inverse diagonal blocks Y_i = L_ii^-T given, row i of the forward sweep is
//   r_i = b_i - sum_{j < i} L_ij x_j,   x_i = Y_i^T r_i
// (backward: columns instead of rows, Y_i instead of its transpose, descending).  The chain
// x_{i-1} -> r_i -> x_i is serial; everything else streams L once.  One CTA a row cannot
// do the chain: it reads 0.75 MB a row by itself (20 us for 256 x 256 doubles).  So:
//   chain  one cluster of BSZ / 32 CTAs; each keeps 32 rows (columns) of the chain.  Per
//          row it takes the block next to the diagonal and the diagonal block itself: its
//          32-row slices arrive by bulk copies into a ring, are held in registers before
//          the vector they wait for is there, and r_i and x_i travel between the CTAs'
//          shared memories (st.async, counted by mbarriers): two exchanges a row.
//   bulk   the other CTAs: each owns slices of 32 rows round robin and takes the published
//          x_j off them, column by column, streaming the slices through the same ring
//          ahead of the vectors.  A slice whose last column outside the band is in goes
//          to the chain.
// Every sum has a fixed order (columns in order, lanes in a tree), so results are bitwise
// reproducible.  x and r travel between chain and bulk through global memory as 16-byte
// pairs (value, the sweep's epoch), stored and read whole: no fence, and a reader's poll
// already has the value.  Every wait is bounded (kWaitClk from when all CTAs are resident): on expiry *err = 2 and the sweep
// winds down.
//
// Measured a sweep (the kernel before: one CTA a row, chain through global flags): FP64
// N=4096 (bsz 128) 208 -> 49.5 us, N=16384 (bsz 256) 1330 -> 184 us (HBM alone: 164 us),
// N=32768 629 us; FP32 factor, N=3000 (bsz 128) 176 -> 39 us, N=32768 1290 -> 445 us.  It
// is bound by the chain (1.5 us a row of 128, 2.1 us of 256) up to about N=10000 and by
// memory above.
#include <cuda.h>
#include <cudaTypedefs.h>

#include "hs_internal.cuh"
#include "hs_mixed.cuh"
#include "stream_common.cuh"

namespace hs {
namespace {

constexpr int kCompute = 256;             // 8 compute warps, 4 rows of a slice each
constexpr int kThreads = kCompute + 96;   // + copies, x in, r in
// blocks before the diagonal that the chain takes itself; the bulk CTAs' sums come back
// within that many steps (2 and 3 blocks, more for the chain to read: N=4096, bsz 128:
// 49.5 -> 57.7 -> 66 us a sweep; N=16384, bsz 256: 184 -> 187 -> 203 us)
constexpr int kBand = 1;
constexpr long long kSettleClk = 100000;  // far longer than a store to another CTA of the cluster takes
constexpr int kSlots = 3;  // x vectors kept (chain: kBand + 1, bulk: 3)

struct SweepArgs {
    const void* L;
    const void* Y;
    const double* in;
    double* out;
    ulonglong2* x;  // nb BSZ pairs: x from the chain to the bulk CTAs
    ulonglong2* r;  // nb BSZ pairs: right-hand sides from the bulk CTAs to the chain
    int* err;
    unsigned* resident;  // two counters of resident CTAs, by the epoch's parity
    int nb;
    unsigned long long epoch;
};

template <int BSZ, typename T>
struct Cfg {
    static constexpr int kRanks = BSZ / 32;
    static constexpr int kTile = 32 * BSZ * (int)sizeof(T);  // a slice of a block
    static constexpr int kStages = kTile >= 65536 ? 3 : (kTile >= 32768 ? 6 : 8);
    static constexpr size_t smem(int slices) {
        return 1024 + (size_t)kStages * kTile + (size_t)(kSlots + 1) * BSZ * 8 + 64 * 8 + 512 + (size_t)slices * 32 * 8;
    }
};

__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ uint32_t map_shared(uint32_t addr, unsigned rank) {
    uint32_t r;
    asm volatile("mapa.shared::cluster.u32 %0, %1, %2;" : "=r"(r) : "r"(addr), "r"(rank));
    return r;
}
// 8 bytes into another CTA's shared memory, counted by the mbarrier beside them
__device__ __forceinline__ void st_async(uint32_t addr, double v, uint32_t bar) {
    asm volatile("st.async.shared::cluster.mbarrier::complete_tx::bytes.b64 [%0], %1, [%2];" ::"r"(addr),
                 "l"(__double_as_longlong(v)), "r"(bar)
                 : "memory");
}
__device__ __forceinline__ void cluster_sync_all() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
// FWD: step t is block row t, off-diagonal slices are rows of L, the diagonal block's are
// columns of Y.  Backward: step t is block row nb-1-t, columns of L and rows of Y.
template <int BSZ, typename T, bool FWD>
__global__ void __launch_bounds__(kThreads, 1)
    sweep_kernel(const __grid_constant__ CUtensorMap mCols, SweepArgs a) {
    using C = Cfg<BSZ, T>;
    constexpr int R = C::kRanks, S = C::kStages;
    using Off = Slice<BSZ, T, !FWD>;
    using Diag = Slice<BSZ, T, FWD>;
    extern __shared__ uint8_t sweep_smem[];
    // the ring starts at the same offset in every CTA of the cluster
    uint8_t* ring = sweep_smem + ((1024u - (smem_u32(sweep_smem) & 1023u)) & 1023u);
    double* xs = reinterpret_cast<double*>(ring + (size_t)S * C::kTile);  // x vectors, [slot][BSZ]
    double* rv = xs + kSlots * BSZ;                                       // chain: r of the step
    double* rslot = rv + BSZ;                                             // chain: the bulk's part of r, [2][32]
    uint64_t* full = reinterpret_cast<uint64_t*>(rslot + 64);
    uint64_t* empty = full + S;
    uint64_t* xbar = empty + S;   // chain: x of the step is complete; bulk: [3] x slot loaded
    uint64_t* xfree = xbar + 3;   // bulk: [3] x slot read
    uint64_t* rbar = xfree + 3;   // chain: r of the step is complete
    uint64_t* rrdy = rbar + 1;    // chain: [2] rslot filled
    uint64_t* rfree = rrdy + 2;   // chain: [2] rslot read
    double* acc = rslot + 64 + 64;  // bulk: running right-hand sides, [slice][32]
    __shared__ ResidentWaits s_waits;
    volatile ResidentWaits* waits = &s_waits;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const unsigned rank = cluster_rank();
    const bool chain = blockIdx.x < R;
    const int nb = a.nb;
    constexpr int band = kBand;
    const size_t bb = (size_t)BSZ * BSZ;
    const T* L = static_cast<const T*>(a.L);
    const T* Y = static_cast<const T*>(a.Y);
    auto row_of = [&](int t) { return FWD ? t : nb - 1 - t; };

    if (tid == 0) {
        for (int i = 0; i < S; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 8);
        }
        for (int i = 0; i < 3; ++i) {
            mbar_init(&xbar[i], 1);
            mbar_init(&xfree[i], 8);
        }
        mbar_init(rbar, 1);
        for (int i = 0; i < 2; ++i) {
            mbar_init(&rrdy[i], 1);
            mbar_init(&rfree[i], 8);
        }
        fence_barrier_init();
        s_waits.fail = 0;
        s_waits.limit = kWaitClk;
        s_waits.resident = a.resident + (a.epoch & 1);
        s_waits.ctas = (int)gridDim.x;
        if (chain) {
            mbar_arrive_expect_tx(&xbar[0], BSZ * 8);
            mbar_arrive_expect_tx(rbar, BSZ * 8);
        }
    }
    // bulk CTA c of P owns slices g = c, c + P, .. of the (nb - band - 1) R slices of the
    // steps after the first band + 1, slice g = step band + 1 + g / R, rows 32 (g % R) ..
    const int P = (int)gridDim.x - R, c = (int)blockIdx.x - R;
    const int nsl = nb > band + 1 ? (nb - band - 1) * R : 0;
    const int own = chain || c >= nsl ? 0 : (nsl - c + P - 1) / P;
    for (int e = tid; e < own * 32; e += kThreads) {
        const int g = c + (e / 32) * P;
        acc[e] = a.in[(size_t)row_of(band + 1 + g / R) * BSZ + 32 * (g % R) + e % 32];
    }
    __syncthreads();
    cluster_sync_all();  // every CTA's barriers are set up
    // the CTAs count themselves in (after the barrier, whose release would wait for it); the next
    // sweep's counter starts at zero
    if (tid == kThreads - 1) {
        atomicAdd(a.resident + (a.epoch & 1), 1u);
        if (blockIdx.x == 0) a.resident[~a.epoch & 1] = 0;
    }

    // the slice `q` of the off-diagonal block of (step t, step s < t), or of Y of step t
    auto copy = [&](uint32_t n, int t, int s, int q) {
        uint8_t* dst = ring + (size_t)(n % S) * C::kTile;
        uint64_t* bar = &full[n % S];
        const int i = row_of(t);
        const bool diag = s == t;
        mbar_arrive_expect_tx(bar, C::kTile);
        if (diag == FWD) {  // columns
            constexpr int kBox = 128 / (int)sizeof(T);
            const int blk = diag ? i : (int)block_id(row_of(s), i, nb);
            for (int h = 0; h < 32 / kBox; ++h)
                tma_load_3d(dst + (size_t)h * BSZ * 128, &mCols, bar, 32 * q + h * kBox, 0, blk);
        } else {
            const T* src = diag ? Y + (size_t)i * bb : L + (size_t)block_id(i, row_of(s), nb) * bb;
            bulk_load(dst, src + (size_t)32 * q * BSZ, C::kTile, bar);
        }
    };

    if (warp == 8) {
        // ---- copies
        if (lane == 0) {
            uint32_t n = 0;
            bool ok = true;
            auto put = [&](int t, int s, int q) {
                if (n >= (uint32_t)S) ok = thread_wait(&empty[n % S], (n / S - 1) & 1, waits);
                if (ok) {
                    copy(n, t, s, q);
                    ++n;
                }
            };
            if (chain) {
                for (int t = 0; t < nb && ok; ++t)
                    for (int s = t > band ? t - band : 0; s <= t && ok; ++s) put(t, s, (int)rank);
            } else {
                for (int s = 0; s < nb - band - 1 && ok; ++s) {
                    // owned slices of steps t >= s + band + 1
                    int e = s * R > c ? (s * R - c + P - 1) / P : 0;
                    for (; e < own && ok; ++e) {
                        const int g = c + e * P;
                        put(band + 1 + g / R, s, g % R);
                    }
                }
            }
            // no copy may still be writing when the CTA leaves
            for (uint32_t h = n > (uint32_t)S ? n - S : 0; h < n; ++h)
                landed(&full[h % S], (h / S) & 1, waits);
        }
        __syncwarp();
    } else if (warp == 9) {
        // ---- bulk: brings x in, steps 0 .. (the last slice's step) - band - 1
        if (own > 0) {
            const int last = (c + (own - 1) * P) / R;
            for (int s = 0; s <= last; ++s) {
                double v[BSZ / 32];
                if (s >= 3 && !warp_wait(&xfree[s % 3], (s / 3 - 1) & 1, waits)) break;
                if (!warp_pairs(a.x + (size_t)s * BSZ, a.epoch, lane, waits, a.err, v)) break;
#pragma unroll
                for (int q = 0; q < BSZ / 32; ++q) xs[(s % 3) * BSZ + lane + 32 * q] = v[q];
                __syncwarp();
                if (lane == 0) mbar_arrive(&xbar[s % 3]);
            }
        }
    } else if (warp == 10) {
        // ---- chain: this CTA's 32 rows of the right-hand side, from the bulk CTAs after
        // the first band + 1 steps
        if (chain) {
            for (int t = 0; t < nb; ++t) {
                if (t >= 2 && !warp_wait(&rfree[t & 1], (t / 2 - 1) & 1, waits)) break;
                double v[1];
                if (t > band) {
                    if (!warp_pairs(a.r + (size_t)t * BSZ + 32 * rank, a.epoch, lane, waits, a.err, v)) break;
                } else {
                    v[0] = a.in[(size_t)row_of(t) * BSZ + 32 * rank + lane];
                }
                rslot[(t & 1) * 32 + lane] = v[0];
                __syncwarp();
                if (lane == 0) mbar_arrive(&rrdy[t & 1]);
            }
        }
    } else if (chain) {
        // ---- chain, 8 warps: outputs 4 warp + lane / 8 of this CTA's 32, sent by lane % 8
        // = the receiving CTA
        const int o = 4 * warp + (lane >> 3), dst = lane & 7;
        uint32_t r_rv = 0, r_xs = 0, r_rbar = 0, r_xbar = 0;
        if (dst < R) {
            r_rv = map_shared(smem_u32(rv + 32 * rank + o), dst);
            r_xs = map_shared(smem_u32(xs + 32 * rank + o), dst);
            r_rbar = map_shared(smem_u32(rbar), dst);
            r_xbar = map_shared(smem_u32(xbar), dst);
        }
        uint32_t n = 0;
        bool ok = true;
        T v[BSZ / 8];
        auto take = [&](auto slice) {  // the next tile into registers, its stage free again
            ok = ok && warp_wait(&full[n % S], (n / S) & 1, waits);
            if (ok) decltype(slice)::load(ring + (size_t)(n % S) * C::kTile, warp, lane, v);
            __syncwarp();
            if (lane == 0) mbar_arrive(&empty[n % S]);
            ++n;
        };
        for (int t = 0; t < nb && ok; ++t) {
            double s4[4] = {0.0, 0.0, 0.0, 0.0};
            for (int s = t > band ? t - band : 0; s < t && ok; ++s) {
                take(Off{});
                // x of the last step is the one still under way; those before it are known
                if (s == t - 1) ok = ok && warp_wait(xbar, s & 1, waits);
                if (!ok) break;
                if (s == t - 1 && tid == 0) mbar_arrive_expect_tx(xbar, BSZ * 8);  // the next phase
                Off::apply(v, xs + (s % (band + 1)) * BSZ, lane, s4);
            }
            ok = ok && warp_wait(&rrdy[t & 1], (t / 2) & 1, waits);
            if (!ok) break;
            const double r = rslot[(t & 1) * 32 + o] - Off::total(s4, lane);
            __syncwarp();
            if (lane == 0) mbar_arrive(&rfree[t & 1]);
            if (dst < R) st_async(r_rv, r, r_rbar);
            take(Diag{});
            ok = ok && warp_wait(rbar, t & 1, waits);
            if (!ok) break;
            if (tid == 0 && t + 1 < nb) mbar_arrive_expect_tx(rbar, BSZ * 8);
            double d4[4] = {0.0, 0.0, 0.0, 0.0};
            Diag::apply(v, rv, lane, d4);
            const double x = Diag::total(d4, lane);
            if (dst < R) st_async(r_xs + (uint32_t)((t % (band + 1)) * BSZ * 8), x, r_xbar);
            if (dst == 0) {
                if (t + band + 1 < nb) pair_store(a.x + (size_t)t * BSZ + 32 * rank + o, x, a.epoch);
                a.out[(size_t)row_of(t) * BSZ + 32 * rank + o] = x;
            }
        }
        // every exchange has landed before this CTA leaves (bounded)
        if (ok) warp_wait(xbar, (nb - 1) & 1, waits);
    } else if (own > 0) {
        // ---- bulk, 8 warps
        const int o = 4 * warp + (lane >> 3);
        uint32_t n = 0;
        bool ok = true;
        const int last = (c + (own - 1) * P) / R;
        for (int s = 0; s <= last && ok; ++s) {
            bool have = false;
            int e = s * R > c ? (s * R - c + P - 1) / P : 0;
            for (; e < own && ok; ++e, ++n) {
                const int g = c + e * P, t = band + 1 + g / R;
                T v[BSZ / 8];
                ok = warp_wait(&full[n % S], (n / S) & 1, waits);
                if (!ok) break;
                Off::load(ring + (size_t)(n % S) * C::kTile, warp, lane, v);
                __syncwarp();
                if (lane == 0) mbar_arrive(&empty[n % S]);
                if (!have && !(ok = warp_wait(&xbar[s % 3], (s / 3) & 1, waits))) break;
                have = true;
                double s4[4] = {0.0, 0.0, 0.0, 0.0};
                Off::apply(v, xs + (s % 3) * BSZ, lane, s4);
                const double tot = Off::total(s4, lane);
                if ((lane & 7) == 0) {
                    const double r = acc[e * 32 + o] - tot;
                    if (s + band + 1 < t)
                        acc[e * 32 + o] = r;
                    else
                        pair_store(a.r + (size_t)t * BSZ + 32 * (g % R) + o, r, a.epoch);
                }
            }
            if (!ok) break;
            if (!have && !(ok = warp_wait(&xbar[s % 3], (s / 3) & 1, waits))) break;
            __syncwarp();
            if (lane == 0) mbar_arrive(&xfree[s % 3]);
        }
    }
    __syncthreads();
    if (tid == 0 && s_waits.fail) atomicExch(a.err, 2);
    cluster_sync_all();  // no CTA leaves while a peer may still write into its memory
    // after a wait ran out, peers' values may be on their way that nothing here has counted
    if (s_waits.fail)
        for (const long long t0 = clock64(); clock64() - t0 < kSettleClk;) {}
}

// columns of 128 bytes, all BSZ rows of a block
template <typename T>
hs_status cols_map(CUtensorMap* m, const T* base, int bsz, int64_t blocks) {
    PFN_cuTensorMapEncodeTiled_v12000 encode = nullptr;
    hs_status st = tensor_map_encoder(&encode);
    if (st != HS_OK) return st;
    cuuint64_t dims[3] = {(cuuint64_t)bsz, (cuuint64_t)bsz, (cuuint64_t)blocks};
    cuuint64_t strides[2] = {(cuuint64_t)bsz * sizeof(T), (cuuint64_t)bsz * bsz * sizeof(T)};
    cuuint32_t box[3] = {(cuuint32_t)(128 / sizeof(T)), (cuuint32_t)bsz, 1};
    cuuint32_t estr[3] = {1, 1, 1};
    const CUresult r = encode(m, sizeof(T) == 8 ? CU_TENSOR_MAP_DATA_TYPE_FLOAT64 : CU_TENSOR_MAP_DATA_TYPE_FLOAT32, 3,
                              const_cast<T*>(base), dims, strides, box, estr, CU_TENSOR_MAP_INTERLEAVE_NONE,
                              CU_TENSOR_MAP_SWIZZLE_128B, CU_TENSOR_MAP_L2_PROMOTION_L2_256B,
                              CU_TENSOR_MAP_FLOAT_OOB_FILL_NONE);
    if (r != CUDA_SUCCESS) {
        set_error("cuTensorMapEncodeTiled failed (" + std::to_string((int)r) + ")");
        return HS_ERR_CUDA;
    }
    return HS_OK;
}

template <int BSZ, typename T, bool FWD>
hs_status launch_dir(hs_ctx ctx, const T* L, const T* Y, const double* in, double* out, unsigned epoch, void* ws,
                     int* err, cudaStream_t s) {
    using C = Cfg<BSZ, T>;
    const int nb = ctx->nb, R = C::kRanks;
    SweepArgs a{};
    a.L = L;
    a.Y = Y;
    a.in = in;
    a.out = out;
    a.x = static_cast<ulonglong2*>(ws);
    a.r = a.x + (size_t)nb * BSZ;
    a.err = err;
    a.resident = reinterpret_cast<unsigned*>(a.r + (size_t)nb * BSZ);
    a.nb = nb;
    a.epoch = epoch;
    CUtensorMap m;
    hs_status st = cols_map<T>(&m, FWD ? Y : L, BSZ, FWD ? (int64_t)nb : total_blocks(nb));
    if (st != HS_OK) return st;
    auto* fn = sweep_kernel<BSZ, T, FWD>;
    cudaLaunchConfig_t cfg{};
    cfg.blockDim = dim3(kThreads);
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = R;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = 1;
    const int64_t nsl = nb > kBand + 1 ? (int64_t)(nb - kBand - 1) * R : 0;
    static int max_clusters[64] = {};  // per device, for the largest shared memory the kernel takes
    const int dev = ctx->device;
    constexpr size_t kMaxSmem = 226 * 1024;
    HS_REQUIRE(dev >= 0 && dev < 64, "device index out of range");
    if (max_clusters[dev] == 0) {
        HS_CUDA(cudaFuncSetAttribute(fn, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kMaxSmem));
        int n = 0;
        cfg.gridDim = dim3(R);
        cfg.dynamicSmemBytes = kMaxSmem;
        HS_CUDA(cudaOccupancyMaxActiveClusters(&n, fn, &cfg));
        HS_REQUIRE(n >= 2, "the sweep needs two resident clusters");
        max_clusters[dev] = n;
    }
    int clusters = max_clusters[dev];
    if ((nsl + R - 1) / R + 1 < clusters) clusters = (int)((nsl + R - 1) / R) + 1;
    const int P = (clusters - 1) * R;
    const int slices = P > 0 ? (int)((nsl + P - 1) / P) : 0;
    cfg.gridDim = dim3(clusters * R);
    cfg.dynamicSmemBytes = C::smem(slices);
    HS_REQUIRE(cfg.dynamicSmemBytes <= kMaxSmem, "matrix too large for the single-launch sweep");
    prof_begin(ctx, s, HS_KERNEL_COLUPD);
    ctx->launches += 1;
    HS_CUDA(cudaLaunchKernelEx(&cfg, fn, m, a));
    const double Tb = (double)nb * (nb - 1) / 2.0;
    prof_end(ctx, s, HS_KERNEL_COLUPD, 2.0 * (Tb + nb) * BSZ * BSZ, (Tb + nb) * sizeof(T) * BSZ * BSZ);
    return HS_OK;
}

template <typename T>
hs_status launch_sweep(hs_ctx ctx, const T* L, const T* Y, const double* in, double* out, int forward, unsigned epoch,
                       void* ws, int* err, cudaStream_t s) {
    const int bsz = ctx->bsz;
    HS_REQUIRE(bsz == 128 || bsz == 256, "the single-launch sweep supports matrixBlockSize 128 or 256");
    if (bsz == 256)
        return forward ? launch_dir<256, T, true>(ctx, L, Y, in, out, epoch, ws, err, s)
                       : launch_dir<256, T, false>(ctx, L, Y, in, out, epoch, ws, err, s);
    return forward ? launch_dir<128, T, true>(ctx, L, Y, in, out, epoch, ws, err, s)
                   : launch_dir<128, T, false>(ctx, L, Y, in, out, epoch, ws, err, s);
}

}  // namespace

size_t sweep_workspace_bytes(int nb, int bsz) {
    return (size_t)2 * nb * bsz * sizeof(ulonglong2) + 256;  // pairs, CTA counters
}

hs_status sweep_reset(hs_ctx ctx, void* ws, cudaStream_t s) {
    HS_CUDA(cudaMemsetAsync(ws, 0, sweep_workspace_bytes(ctx->nb, ctx->bsz), s));
    return HS_OK;
}

hs_status launch_sweep_f32(hs_ctx ctx, const float* L, const float* Y, const double* in, double* out, int forward,
                           unsigned epoch, void* ws, int* err, cudaStream_t s) {
    return launch_sweep<float>(ctx, L, Y, in, out, forward, epoch, ws, err, s);
}

hs_status launch_sweep_f64(hs_ctx ctx, const double* L, const double* Y, const double* in, double* out, int forward,
                           unsigned epoch, void* ws, int* err, cudaStream_t s) {
    return launch_sweep<double>(ctx, L, Y, in, out, forward, epoch, ws, err, s);
}

}  // namespace hs
