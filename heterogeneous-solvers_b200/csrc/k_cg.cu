// k_cg.cu — conjugate gradients on the packed symmetric matrix, a run of iterations in one
// persistent launch.
//
// Reference path replaced: CG.cpp:38-163, 277-528 (block sizes 128 and 256; other sizes and
// the reference-order mode run the launch-per-operation driver in hs_solvers.cu).
//
// An iteration is two phases with a grid-wide sum between them:
//   A   q = A d as partial sums.  The stored blocks in packed order are one array of units
//       of 4 KB (4 rows of 128, 2 of 256); every CTA owns a contiguous range of them, its
//       warps take turns, and each streams its units through three stages of its own by
//       bulk copies that run on across phases and iterations (up to three units a warp
//       stay there).  A unit is applied as it is (rows of q, kept per block) and transposed
//       (summed over the range's units of a block column, in registers and then over the
//       warps).  d = r + beta d is formed where it is read.  The CTA's part of d.q comes
//       along.
//   sum d.q -> alpha
//   B   each 32 elements of q from their partial sums in a fixed order; x += alpha d,
//       r -= alpha q, the new d stored for the next iteration; part of r.r
//   sum r.r -> beta
// Every 50th iteration recomputes r = b - A x with a second pass, as the reference does.
// The sums are the barriers: a CTA stores its part and counts itself in, and once all are in
// every CTA adds up the parts in order, so all take the same decisions from the same bits,
// and results are bitwise reproducible.  Every wait is bounded; on expiry *err = 1 and the
// launch winds down.  (Slices of 32 rows shared by all warps of a CTA, with warps of their
// own for copies and vectors, took 1 us a slice: every warp's latency was exposed.  Parts
// polled as value-and-epoch pairs by all CTAs cost 8k cycles a sum.)
//
// Measured an iteration, against a launch per operation with two host reads an iteration:
// N=4096 (bsz 128) 57 -> 15 us (7 us the pass over 67 MB, which L2 just does not hold, the
// rest two sums and phase B), N=15000 (bsz 256, 0.9 GB) 200 -> 160 us, of which the pass is
// 145 (6.3 TB/s).
#include <algorithm>

#include "stream_common.cuh"

namespace hs {
namespace {

constexpr int kWarps = 16;
constexpr int kThreads = 32 * kWarps;
constexpr int kUnit = 512;              // doubles: 4 KB
constexpr int kStages = 3;
constexpr int kMaxCtas = 160;           // parts a grid-wide sum reads: 5 a lane

struct CgState {
    double delta, delta_zero, beta;
    long long it;
    unsigned long long sums;  // grid-wide sums so far
    int cur;        // index of the d buffer that holds the last d
    int done;       // converged (or not a number)
};

struct CgArgs {
    const double* A;
    const double* b;
    double *x, *r, *d;   // d: two buffers of n
    double *prow, *pcol; // partial sums: [block row][block column][row], [CTA + column][row]
    double* parts;       // [2][CTA]
    unsigned long long* count;  // CTAs counted in, over all sums
    CgState* state;
    int* err;
    int nb;
    unsigned units;
    long long it_end;    // iterations after which this launch stops
    double eps2;
    int first;           // the initial residual first
};

template <int BSZ>
constexpr size_t cg_smem_bytes() {
    return 1024 + (size_t)kWarps * (kStages * kUnit + BSZ) * 8;
}

// the first unit of range w of W, and the range of a unit
__device__ __forceinline__ unsigned range_start(unsigned total, unsigned W, unsigned w) {
    const unsigned base = total / W, rem = total % W;
    return w * base + (w < rem ? w : rem);
}
__device__ __forceinline__ unsigned range_owner(unsigned base, unsigned rem, unsigned u) {
    const unsigned cut = rem * (base + 1);
    return u < cut ? u / (base + 1) : rem + (u - cut) / base;
}

template <int BSZ>
__global__ void __launch_bounds__(kThreads, 1) cg_kernel(CgArgs a) {
    constexpr int RW = kUnit / BSZ;        // rows of a unit
    constexpr unsigned UB = BSZ / RW;      // units of a block
    constexpr int NC = BSZ / 32;           // columns a lane has: (m * 32 + lane) * 2 + {0, 1}
    extern __shared__ uint8_t cg_smem[];
    double* ring = reinterpret_cast<double*>(cg_smem + ((1024u - (smem_u32(cg_smem) & 1023u)) & 1023u));
    double* red = ring + kWarps * kStages * kUnit;  // [warp][BSZ]
    __shared__ uint64_t s_full[kWarps][kStages], s_read[kWarps][kStages];
    __shared__ double s_rows[kWarps][2][RW], s_part[kWarps], s_sum;
    __shared__ Waits s_waits;
    __shared__ int s_good;
    volatile Waits* waits = &s_waits;

    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    const int P = gridDim.x, c = blockIdx.x, nb = a.nb;
    const int64_t n = (int64_t)nb * BSZ;
    const unsigned rbase = a.units / P, rrem = a.units % P;
    const unsigned lo = range_start(a.units, P, c), hi = range_start(a.units, P, c + 1);
    auto column_unit = [&](int j) { return (unsigned)column_start(j, nb) * UB; };
    int ja, jb, unused;  // the range's block columns; its part of column j: [seg_lo(j), seg_hi(j))
    block_coords(lo / UB, nb, &unused, &ja);
    block_coords((hi - 1) / UB, nb, &unused, &jb);
    auto seg_lo = [&](int j) { return j == ja ? lo : column_unit(j); };
    auto seg_hi = [&](int j) { return j == jb ? hi : column_unit(j + 1); };
    int own = 0;  // units of this warp
    for (int j = ja; j <= jb; ++j) {
        const int len = (int)(seg_hi(j) - seg_lo(j));
        own += len > warp ? (len - warp + kWarps - 1) / kWarps : 0;
    }
    // copies go on (else the units all stay and are read once, or a wait for one has run out)
    bool streaming = own > kStages;
    double* stage = ring + (size_t)warp * kStages * kUnit;
    uint64_t *full = s_full[warp], *read = s_read[warp];

    if (lane == 0) {
        for (int k = 0; k < kStages; ++k) {
            mbar_init(&full[k], 1);
            mbar_init(&read[k], 1);
        }
        fence_barrier_init();
    }
    if (tid == 0) {
        s_waits.fail = 0;
        s_waits.limit = kWaitClk;
    }
    __syncthreads();
    uint32_t issued = 0, m = 0;  // this warp's copies, and the next of them to be used
    // the unit of the next copy: the warp's units round and round
    int pj = ja;
    unsigned pu = lo + warp, phi = seg_hi(ja);
    auto settle = [&]() {  // (own > 0)
        while (pu >= phi) {
            pj = pj == jb ? ja : pj + 1;
            pu = seg_lo(pj) + warp;
            phi = seg_hi(pj);
        }
    };
    auto copy = [&]() {
        if (lane == 0) {
            uint64_t* bar = &full[issued % kStages];
            mbar_arrive_expect_tx(bar, kUnit * 8);
            bulk_load(stage + (size_t)(issued % kStages) * kUnit, a.A + (size_t)pu * kUnit, kUnit * 8, bar);
        }
        ++issued;
        pu += kWarps;
        settle();
    };
    if (own > 0) settle();
    for (int k = 0; k < kStages && k < own; ++k) copy();

    CgState st = *a.state;
    bool ok = true;
    const double* db[2] = {a.d, a.d + n};

    // sum over all CTAs of v (fixed order), a grid-wide barrier on the way
    auto grid_sum = [&](double v) -> double {
        ++st.sums;
        for (int o = 16; o > 0; o >>= 1) v += __shfl_xor_sync(0xffffffffu, v, o);
        if (lane == 0) s_part[warp] = v;
        __syncthreads();
        if (warp == 0) {
            double* part = a.parts + (size_t)(st.sums & 1) * P;
            double t = lane < kWarps ? s_part[lane] : 0.0;
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) {
                __stcg(part + c, t);
                __threadfence();
                atomicAdd(a.count, 1ull);
            }
            __syncwarp();
            warp_count(a.count, st.sums * (unsigned long long)P, lane, waits);
            double y[kMaxCtas / 32];
#pragma unroll
            for (int k = 0; k < kMaxCtas / 32; ++k) y[k] = lane + 32 * k < P ? __ldcg(part + lane + 32 * k) : 0.0;
            t = 0.0;
#pragma unroll
            for (int k = 0; k < kMaxCtas / 32; ++k) t += y[k];
            for (int o = 16; o > 0; o >>= 1) t += __shfl_xor_sync(0xffffffffu, t, o);
            if (lane == 0) {
                s_sum = t;
                s_good = waits->fail == 0;  // one answer for all warps
                if (!s_good) atomicExch(a.err, 1);
            }
        }
        __syncthreads();
        ok = ok && s_good != 0;
        return s_sum;
    };

    // phase A: partial sums of A v; v = r + beta d (type 0) or x (type 1).  Returns this
    // thread's part of v . A v.  A wait that runs out leaves its mark and the pass goes on
    // to its end without further copies (later waits return at once); the next grid_sum ends
    // the launch.
    auto matvec = [&](int type, double beta, const double* dold) -> double {
        auto val = [&](int64_t e) -> double {
            return type == 0 ? fma(beta, __ldcg(dold + e), __ldcg(a.r + e)) : __ldcg(a.x + e);
        };
        double dq = 0.0;
        if (!streaming) m = 0;  // the units are where they were
        for (int j = ja; j <= jb; ++j) {
            const unsigned u0 = column_unit(j), uhi = seg_hi(j);
            // the rows of v of a unit, read one unit ahead
            auto rows = [&](unsigned u) -> double {
                return lane < RW && u < uhi ? val((int64_t)j * BSZ + (int64_t)(u - u0) * RW + lane) : 0.0;
            };
            unsigned u = seg_lo(j) + warp;
            double rv = rows(u);
            double xj[NC], ca[NC];
#pragma unroll
            for (int e = 0; e < NC; ++e) {
                ca[e] = 0.0;
                xj[e] = val((int64_t)j * BSZ + (e / 2 * 32 + lane) * 2 + (e & 1));
            }
            for (; u < uhi; u += kWarps, ++m) {
                streaming &= warp_wait(&full[m % kStages], (m / kStages) & 1, waits);
                double* vr = s_rows[warp][m & 1];
                if (lane < RW) vr[lane] = rv;
                rv = rows(u + kWarps);
                double v[RW * NC];
                const double* src = stage + (size_t)(m % kStages) * kUnit + 2 * lane;
#pragma unroll
                for (int e = 0; e < RW * NC; e += 2) {
                    const double2 t = *reinterpret_cast<const double2*>(src + 32 * e);
                    v[e] = t.x;
                    v[e + 1] = t.y;
                }
                __syncwarp();
                // The stage is refilled through an mbarrier that this warp itself completes: an
                // arrival follows the reads before it.  (Ordered by __syncwarp alone, the
                // copy's write overtook reads still queued, once in some 10^8 units.)
                if (lane == 0) mbar_arrive(&read[m % kStages]);
                // v[r NC + e]: row r, the lane's column e
                const unsigned off = u - u0;
                const bool diag = off < UB;
                double s[RW];
#pragma unroll
                for (int r = 0; r < RW; ++r) {
                    s[r] = 0.0;
#pragma unroll
                    for (int e = 0; e < NC; ++e) s[r] = fma(v[r * NC + e], xj[e], s[r]);
                    const double d = diag ? 0.0 : vr[r];
#pragma unroll
                    for (int e = 0; e < NC; ++e) ca[e] = fma(v[r * NC + e], d, ca[e]);
                }
                // row totals: row lane / (32 / RW)
                const bool b4 = lane & 16, b3 = lane & 8;
                double t;
                if constexpr (RW == 4) {
                    const double g0 = (b4 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, b4 ? s[0] : s[2], 16);
                    const double g1 = (b4 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, b4 ? s[1] : s[3], 16);
                    t = (b3 ? g1 : g0) + __shfl_xor_sync(0xffffffffu, b3 ? g0 : g1, 8);
                } else {
                    t = (b4 ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, b4 ? s[0] : s[1], 16);
                    t += __shfl_xor_sync(0xffffffffu, t, 8);
                }
                t += __shfl_xor_sync(0xffffffffu, t, 4);
                t += __shfl_xor_sync(0xffffffffu, t, 2);
                t += __shfl_xor_sync(0xffffffffu, t, 1);
                // Only what has been read may be overwritten.  (The reads are long done here.  A
                // refill before the totals is 1 % faster from L2 and slower from HBM: N = 131072
                // 11.45 against 10.85 ms an iteration.)
                if (streaming) {
                    streaming = warp_wait(&read[m % kStages], (m / kStages) & 1, waits);
                    if (streaming) copy();
                }
                if (lane % (32 / RW) == 0) {
                    const int r = lane / (32 / RW), i = j + (int)(off / UB);
                    __stcg(a.prow + ((size_t)i * (i + 1) / 2 + j) * BSZ + (off % UB) * RW + r, t);
                    dq = fma(diag ? vr[r] : 2.0 * vr[r], t, dq);
                }
            }
            // the column's transposed sums over the warps
#pragma unroll
            for (int e = 0; e < NC; e += 2)
                *reinterpret_cast<double2*>(red + warp * BSZ + (e / 2 * 32 + lane) * 2) = make_double2(ca[e], ca[e + 1]);
            __syncthreads();
            if (tid < BSZ) {
                double t = 0.0;
#pragma unroll
                for (int w = 0; w < kWarps; ++w) t += red[w * BSZ + tid];
                __stcg(a.pcol + ((size_t)c + j) * BSZ + tid, t);
            }
            __syncthreads();
        }
        return dq;
    };

    // phase B: element e's sum, for 32 elements a step: before(e) and after(e, sum) by warp
    // 0's lanes
    auto reduce = [&](auto before, auto after) {
        for (long long ch = c; ch < n / 32; ch += P) {
            const int i = (int)(ch * 32 / BSZ), r = (int)(ch * 32 % BSZ) + lane;
            if (warp == 0) before(ch * 32 + lane);
            const double* p = a.prow + (size_t)i * (i + 1) / 2 * BSZ + r;
            // transposed parts: the CTAs whose ranges meet block column i
            const unsigned k0 = range_owner(rbase, rrem, column_unit(i));
            const unsigned k1 = range_owner(rbase, rrem, column_unit(i + 1) - 1);
            const double* pc = a.pcol + ((size_t)k0 + i) * BSZ + r;
            // both lists as one, 8 loads of a warp in flight at a time
            const int nr = i + 1, total = nr + (int)(k1 - k0) + 1;
            double t = 0.0;
            for (int m0 = warp; m0 < total; m0 += 8 * kWarps) {
                double y[8];
#pragma unroll
                for (int h = 0; h < 8; ++h) {
                    const int m = m0 + h * kWarps;
                    y[h] = m < total ? __ldcg(m < nr ? p + (size_t)m * BSZ : pc + (size_t)(m - nr) * BSZ) : 0.0;
                }
#pragma unroll
                for (int h = 0; h < 8; ++h) t += y[h];
            }
            red[warp * 32 + lane] = t;
            __syncthreads();
            if (warp == 0) {
                t = 0.0;
#pragma unroll
                for (int k = 0; k < kWarps; ++k) t += red[k * 32 + lane];
                after(ch * 32 + lane, t);
            }
            __syncthreads();
        }
    };

    double eb = 0.0, er = 0.0, ed = 0.0, ex = 0.0;  // an element's entries, read ahead of its sum
    auto read_b = [&](long long e) { eb = a.b[e]; };
    if (a.first) {
        // r = b - A x
        matvec(1, 0.0, nullptr);
        grid_sum(0.0);
        double rr = 0.0;
        if (ok)
            reduce(read_b, [&](long long e, double q) {
                const double r = eb - q;
                __stcg(a.r + e, r);
                rr = fma(r, r, rr);
            });
        st.delta = st.delta_zero = grid_sum(rr);
        st.beta = 0.0;
        st.it = 0;
        st.cur = 0;
    }
    // (a comparison that a NaN ends, as the reference's loop condition)
    while (ok && st.it < a.it_end && st.delta > a.eps2 * st.delta_zero) {
        const double* dold = db[st.cur];
        double* dnew = const_cast<double*>(db[st.cur ^ 1]);
        const double dq = grid_sum(matvec(0, st.beta, dold));
        if (!ok) break;
        const double alpha = st.delta / dq;
        const bool recompute = st.it % 50 == 0;
        double rr = 0.0;
        reduce(
            [&](long long e) {
                er = __ldcg(a.r + e);
                ed = __ldcg(dold + e);
                ex = __ldcg(a.x + e);
            },
            [&](long long e, double q) {
                const double d = fma(st.beta, ed, er);
                __stcg(dnew + e, d);
                __stcg(a.x + e, fma(d, alpha, ex));
                if (!recompute) {
                    const double rn = fma(-alpha, q, er);
                    __stcg(a.r + e, rn);
                    rr = fma(rn, rn, rr);
                }
            });
        if (recompute) {
            grid_sum(0.0);
            if (!ok) break;
            matvec(1, 0.0, nullptr);
            grid_sum(0.0);
            if (!ok) break;
            reduce(read_b, [&](long long e, double q) {
                const double rn = eb - q;
                __stcg(a.r + e, rn);
                rr = fma(rn, rn, rr);
            });
        }
        const double delta = grid_sum(rr);
        st.beta = delta / st.delta;
        st.delta = delta;
        st.cur ^= 1;
        ++st.it;
    }
    if (c == 0 && tid == 0) {
        st.done = !(st.delta > a.eps2 * st.delta_zero);
        *a.state = st;
    }
    // no copy may still be writing when the CTA leaves
    for (uint32_t h = issued > (uint32_t)kStages ? issued - kStages : 0; h < issued; ++h)
        landed(&full[h % kStages], (h / kStages) & 1, waits);
    __syncthreads();
    if (tid == 0 && s_waits.fail) atomicExch(a.err, 1);
}

template <int BSZ>
hs_status run(hs_ctx ctx, CgArgs a, int grid, cudaStream_t s) {
    static bool attr[64] = {};
    if (ctx->device < 0 || ctx->device >= 64 || !attr[ctx->device]) {
        HS_CUDA(cudaFuncSetAttribute(cg_kernel<BSZ>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)cg_smem_bytes<BSZ>()));
        if (ctx->device >= 0 && ctx->device < 64) attr[ctx->device] = true;
    }
    void* args[] = {&a};
    ctx->launches += 1;
    Turn turn(ctx, s);
    if (turn.status != HS_OK) return turn.status;
    // cooperative: the CTAs wait for one another
    HS_CUDA(cudaLaunchCooperativeKernel((const void*)cg_kernel<BSZ>, dim3(grid), dim3(kThreads), args,
                                        cg_smem_bytes<BSZ>(), s));
    return HS_OK;
}

}  // namespace

hs_status cg_persistent(hs_ctx ctx, const double* A, const double* b, double* x, double eps, int64_t imax,
                        int64_t* iters_out, double* dnew_out, double* d0_out) {
    const int nb = ctx->nb, bsz = ctx->bsz;
    HS_REQUIRE(bsz == 128 || bsz == 256, "the persistent CG supports matrixBlockSize 128 or 256");
    HS_REQUIRE(reinterpret_cast<uintptr_t>(A) % 16 == 0, "the matrix must be aligned to 16 bytes");
    cudaStream_t s = ctx->stream;
    const int64_t n = (int64_t)nb * bsz;
    CgArgs a{};
    const int64_t units = total_blocks(nb) * ((int64_t)bsz * bsz / kUnit);
    HS_REQUIRE(units < (1LL << 31), "matrix too large for the persistent CG");
    a.units = (unsigned)units;
    const int grid = (int)std::min<int64_t>(std::min(ctx->num_sms, kMaxCtas), (units + kWarps - 1) / kWarps);
    const size_t prow = (size_t)total_blocks(nb) * bsz, pcol = (size_t)(nb + grid) * bsz;
    hs_status st = ensure_work(ctx, (size_t)3 * n * sizeof(double));
    if (st != HS_OK) return st;
    st = ensure_scratch(ctx, kSmallScratch + (prow + pcol) * sizeof(double) + 2 * (size_t)grid * sizeof(double) + 512);
    if (st != HS_OK) return st;
    a.A = A;
    a.b = b;
    a.x = x;
    a.r = static_cast<double*>(ctx->work);
    a.d = a.r + n;
    a.prow = reinterpret_cast<double*>(static_cast<char*>(ctx->scratch) + kSmallScratch);
    a.pcol = a.prow + prow;
    a.parts = a.pcol + pcol;
    a.state = reinterpret_cast<CgState*>(a.parts + 2 * (size_t)grid);
    a.err = reinterpret_cast<int*>(a.state + 1);
    a.count = reinterpret_cast<unsigned long long*>(a.state + 1) + 16;  // a line of its own
    a.nb = nb;
    a.eps2 = eps * eps;
    if ((st = turn_mark(ctx, s)) != HS_OK || (st = turn_ready(ctx)) != HS_OK) return st;
    HS_CUDA(cudaMemsetAsync(x, 0, n * sizeof(double), s));
    HS_CUDA(cudaMemsetAsync(a.d, 0, 2 * n * sizeof(double), s));
    HS_CUDA(cudaMemsetAsync(a.parts, 0, 2 * (size_t)grid * sizeof(double) + 512, s));
    // a launch runs iterations for about a tenth of a second at most (5e11 bytes of matrix),
    // so that the stream and the host see progress
    const double bytes = (double)total_blocks(nb) * bsz * bsz * 8.0;
    const int64_t chunk = std::max<int64_t>(4, std::min<int64_t>(1000, (int64_t)(5e11 / bytes)));
    struct {
        CgState st;
        int err;
    } h{};
    static_assert(sizeof(CgState) % 4 == 0, "err follows the state");
    volatile char* pinned = reinterpret_cast<volatile char*>(ctx->h_pinned);
    int64_t it0 = 0;
    for (a.first = 1;; a.first = 0) {
        a.it_end = std::min<int64_t>(imax, it0 + chunk);
        prof_begin(ctx, s, HS_KERNEL_SYMV);
        st = bsz == 256 ? run<256>(ctx, a, grid, s) : run<128>(ctx, a, grid, s);
        if (st != HS_OK) return st;
        HS_CUDA(cudaMemcpyAsync((void*)pinned, a.state, sizeof(h), cudaMemcpyDeviceToHost, s));
        HS_CUDA(cudaStreamSynchronize(s));
        std::copy(const_cast<const char*>(reinterpret_cast<volatile char*>(pinned)),
                  const_cast<const char*>(reinterpret_cast<volatile char*>(pinned)) + sizeof(h),
                  reinterpret_cast<char*>(&h));
        // matvec passes of this launch: one an iteration, a second one every 50th, the first residual
        const int64_t passes = (h.st.it - it0) + ((h.st.it + 49) / 50 - (it0 + 49) / 50) + a.first;
        prof_end(ctx, s, HS_KERNEL_SYMV, 2.0 * passes * (double)n * n, passes * (bytes + 24.0 * n));
        if (h.err) {
            set_error("hs_cg_solve: a bounded wait of the persistent iteration ran out");
            return HS_ERR_TIMEOUT;
        }
        it0 = h.st.it;
        if (h.st.done || it0 >= imax) break;
    }
    if (iters_out) *iters_out = it0;
    if (dnew_out) *dnew_out = h.st.delta;
    if (d0_out) *d0_out = h.st.delta_zero;
    if (it0 >= imax && h.st.delta > a.eps2 * h.st.delta_zero) {
        set_error("hs_cg_solve: iMax reached before the tolerance (delta_new = " + std::to_string(h.st.delta) +
                  ", target " + std::to_string(a.eps2 * h.st.delta_zero) + ")");
        return HS_ERR_NO_CONVERGENCE;
    }
    return HS_OK;
}

}  // namespace hs
