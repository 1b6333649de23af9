// k_split_update.cu — the FP64 trailing update on the tensor cores' INT8 path.
//
// The large trailing updates of the FP64 Cholesky (MatrixMatrixOperations.cpp:146-906) are
// C <- C - P P^T with a panel P of one block column, or of two at once; the inverse of the
// likelihood's gradient is built from updates C <- C +- P Q^T of the same form.  The FP64
// tensor pipe bounds them at 64 multiply-adds a cycle and SM; the INT8 pipe does 8192.  Each
// row of a panel is therefore scaled by a power of two to |t| <= 0.497 and written as seven
// balanced base-256 digits, t = sum_i d_i 2^-8(i+1) with |error| <= 2^-57, and the product of
// two rows is the sum over levels l = i + j of 2^-8l (digit plane i) x (digit plane j): exact
// INT32 sums in the tensor cores, levels 0..7 kept (34 plane products), carried into one
// 64-bit integer, rounded to FP64 once and added to C.  (K. Ozaki, T. Ogita, S. Oishi, S. M.
// Rump, "Error-free transformations of matrix multiplication by using fast routines of matrix
// multiplication and its applications", 2012; H. Ootomo, K. Ozaki, R. Yokota, "DGEMM on
// integer matrix multiplication unit", 2024.)
//
// Error of one update, in units of the rows' scales: the digits' 2^-57 a factor, levels
// past 7 at most 1.26 x 2^-64 a product (five products of 2^14 x 2^-80 at level 8) and the
// last unit 2^-57; then a rounding of the product and one of C.  The FP64 pipe's chain rounds
// 64 times at 2^-53 |C|.  Measured, max |A - L L^T| / sqrt(a_ii a_jj) of a factor at N = 4800
// (Wishart): 7.6e-15 -> 2.4e-15.  Scale_i scale_j <= 16.2 max|P_i| max|P_j| <= 16.2 sqrt(A_ii
// A_jj) (a row's scale is at most 4 / 0.994 times its largest entry), so the factor keeps the
// plain form's backward error bound relative to sqrt(A_ii A_jj).  It does not keep the plain
// form's bound by entries, |L| |L|^T: what lies more than 2^-56 below the largest entry of a
// row's panel (of both, where two go at once) does not enter the product.
#include "hs_internal.cuh"
#include "stream_common.cuh"
#include "tc_common.cuh"

namespace hs {

namespace {

using namespace tc;

constexpr int kPlanes = 7, kHighPlanes = 4;  // digits a value; those of levels 0..3
constexpr int kKc = 64;                      // K bytes a stage (64-byte swizzle)
constexpr int kPlane = 128 * kKc;            // one plane of 128 rows of a stage
constexpr int kOperand = kPlanes * kPlane;
constexpr int kStage = 2 * kOperand, kStages = 2;  // 112 KB each
constexpr int kSmem = 512 + kStages * kStage + 256 * 8 + 112;  // + the tile's scales, barriers
constexpr int kEpi = 8, kThreads = 64 + 32 * kEpi;  // copy warp, MMA warp, epilogue warps
constexpr int kPerCta = 4;     // tiles a CTA
constexpr int kMinExp = -900;  // rows whose largest entry lies below 2^-900 keep that scale

// ------------------------------------------------------------------ digits
// One row's scale and seven planes, by a warp whose lane holds entries E lane .. of the K = 32 E,
// in the order the update reads them: for each 128 rows and 64 columns the planes one after
// the other, each as 64-byte rows with the 64-byte swizzle (16-byte unit u of row r at
// u ^ (r / 2 % 4)), so that an operand's stage is one contiguous copy.  A row that holds an
// infinity or NaN gets the scale NaN (and zero digits), so that what it updates becomes NaN.
template <int E>
__device__ __forceinline__ void split_row(const double (&v)[E], int64_t row, int lane, int8_t* D, double* scale) {
    constexpr int K = 32 * E;
    long long m = 0;
#pragma unroll
    for (int q = 0; q < E; ++q) m = max(m, __double_as_longlong(v[q]) & 0x7fffffffffffffffll);
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) m = max(m, __shfl_xor_sync(0xffffffffu, m, o));
    const bool finite = m < 0x7ff0000000000000ll;
    // m < 2^(E - 1022); |t| = |x| 2^-e <= 0.497 keeps every digit within [-128, 127]
    int e = max((int)(m >> 52) - 1021 + (((m >> 44) & 0xff) >= 0xfd), kMinExp);
    const double s = __longlong_as_double((long long)(56 - (finite ? e : 0) + 1023) << 52);
    unsigned long long u[E];
#pragma unroll
    for (int q = 0; q < E; ++q) {
        // adding 128 to every digit makes the bytes of the sum the digits plus 128
        const long long t = finite ? __double2ll_rn(v[q] * s) : 0;
        u[q] = ((unsigned long long)(t + 0x0080808080808080ll)) ^ 0x0080808080808080ull;
    }
    const int r = (int)(row & 127), chunk = lane * E / kKc, byte = lane * E % kKc;
    int8_t* out = D + ((row >> 7) * (K / kKc) + chunk) * kOperand + r * kKc +
                  (((byte >> 4) ^ (r >> 1 & 3)) << 4) + (byte & 15);
#pragma unroll
    for (int i = 0; i < kPlanes; ++i) {
        const int sh = 8 * (kPlanes - 1 - i);
        unsigned w[E / 4];
#pragma unroll
        for (int q = 0; q < E / 4; ++q)
            w[q] = (unsigned)(u[4 * q] >> sh & 0xff) | (unsigned)(u[4 * q + 1] >> sh & 0xff) << 8 |
                   (unsigned)(u[4 * q + 2] >> sh & 0xff) << 16 | (unsigned)(u[4 * q + 3] >> sh & 0xff) << 24;
        int8_t* dst = out + i * kPlane;
        if constexpr (E == 16)
            *reinterpret_cast<uint4*>(dst) = make_uint4(w[0], w[1], w[2], w[3]);
        else
            *reinterpret_cast<uint2*>(dst) = make_uint2(w[0], w[1]);
    }
    // two rows' scales together turn units of 2^-56 into the product
    if (lane == 0)
        scale[row] = finite ? __longlong_as_double((long long)(e - 28 + 1023) << 52) : __longlong_as_double(~0ll);
}

// The rows of a panel; K entries a row: of one panel (P1 unused) or half of them of each of two.
template <int K>
__global__ void __launch_bounds__(256) digits_kernel(const double* __restrict__ P0, const double* __restrict__ P1, int bsz,
                                                     int64_t rows, int8_t* __restrict__ D, double* __restrict__ scale) {
    constexpr int E = K / 32;  // entries a lane
    const int64_t row = (int64_t)blockIdx.x * 8 + (threadIdx.x >> 5);
    const int lane = threadIdx.x & 31;
    if (row >= rows) return;
    const double* src = (lane * E < bsz ? P0 : P1) + row * bsz + lane * E % bsz;
    double v[E];
#pragma unroll
    for (int q = 0; q < E / 2; ++q) {
        const double2 x = *reinterpret_cast<const double2*>(src + 2 * q);
        v[2 * q] = x.x;
        v[2 * q + 1] = x.y;
    }
    split_row<E>(v, row, lane, D, scale);
}

// The columns of consecutive blocks of 256, 16 of them a CTA
__global__ void __launch_bounds__(256) digits_transposed_kernel(const double* __restrict__ P, int8_t* __restrict__ D,
                                                                double* __restrict__ scale) {
    __shared__ double t[256][17];
    const double* src = P + (size_t)blockIdx.y * 65536 + blockIdx.x * 16;
    for (int e = threadIdx.x; e < 256 * 16; e += 256) t[e >> 4][e & 15] = src[(size_t)(e >> 4) * 256 + (e & 15)];
    __syncthreads();
    const int lane = threadIdx.x & 31;
#pragma unroll
    for (int z = 0; z < 2; ++z) {
        const int c = 2 * (threadIdx.x >> 5) + z;
        double v[8];
#pragma unroll
        for (int q = 0; q < 8; ++q) v[q] = t[8 * lane + q][c];
        split_row<8>(v, (int64_t)blockIdx.y * 256 + blockIdx.x * 16 + c, lane, D, scale);
    }
}

// ------------------------------------------------------------------ update
// C += sign A B^T over a part of the blocks of C
struct SplitArgs {
    double* C;
    const int8_t *digA, *digB;
    const double *scaleA, *scaleB;
    double sign;
    int depth;         // columns of A and B: 256 or 512
    int nb, bsz;
    int by_rows;       // C: blocks of a lower triangle stored row by row (else column by column)
    int rows;          // 0: a lower triangle of `cols` block columns; else a rectangle of rows x cols
    int cols;
    int r0, c0;        // its first block row and column in C
    int offset;        // the same in A's and B's digits (in blocks)
    int64_t items;     // 128 x 128 tiles
    long long* info;
};

// kind::i8 instruction descriptor: D s32 (2 at bit 4), A and B signed (1 at bits 7 and 10),
// both K-major, N >> 3 in [17, 23), M >> 4 in [24, 29)
constexpr uint32_t kIdesc = (2u << 4) | (1u << 7) | (1u << 10) | ((128u >> 3) << 17) | ((128u >> 4) << 24);

// the descriptors' low words; the rest is the same for every plane
__device__ __forceinline__ void umma_i8(uint32_t d, uint32_t a, uint32_t b, uint32_t high, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %3};\n\tmov.b64 db, {%2, %3};\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], da, db, %4, p;\n\t}\n" ::"r"(d),
        "r"(a), "r"(b), "r"(high), "r"(kIdesc), "r"(accumulate)
        : "memory");
}

// The products of levels LEVEL + 3 .. LEVEL of one stage, highest first, as straight-line code
// with descriptors at constant distances, issued by one lane of a warp that walks the loop
// together (a product takes the tensor core 35 ns; issued by a lone thread 53 ns, and
// with descriptors formed in a loop 68 ns).  wait / done: the four accumulators' barriers, or
// null.
template <int LEVEL>
__device__ __forceinline__ bool issue_levels(uint32_t taddr, uint64_t desc, uint32_t accumulate, uint64_t* wait,
                                             uint64_t* done, uint32_t parity, bool leader, volatile Waits* waits) {
    const uint32_t da = (uint32_t)desc, db = da + (kOperand >> 4), high = (uint32_t)(desc >> 32);
#pragma unroll
    for (int x = 0; x < 4; ++x) {
        if (wait) {
            if (!suspended_wait_warp(&wait[x], parity, waits)) return false;
            tc_fence_after();
        }
        if (leader) {
            constexpr int kTop = kPlanes - 1;
            const int level = LEVEL + 3 - x, first = level > kTop ? level - kTop : 0, last = level < kTop ? level : kTop;
#pragma unroll
            for (int i = first; i <= last; ++i)
#pragma unroll
                for (int ks = 0; ks < kKc / 32; ++ks)
                    umma_i8(taddr + x * 128, da + ((i * kPlane + ks * 32) >> 4),
                            db + (((level - i) * kPlane + ks * 32) >> 4), high, i > first || ks > 0 ? 1u : accumulate);
            if (done) umma_commit(&done[x]);
        }
        __syncwarp();
    }
    return true;
}

// top 2^32 + low, rounded to nearest; exact halves by the exponent's position (the conversion
// instruction from 64 bits is slower)
__device__ __forceinline__ double to_double(int top, unsigned low) {
    const double hi = __hiloint2double(0x43300000, top ^ (int)0x80000000) - 4503601774854144.0;  // 2^52 + 2^31
    const double lo = __hiloint2double(0x43300000, (int)low) - 4503599627370496.0;               // 2^52
    return fma(hi, 4294967296.0, lo);
}

__device__ __forceinline__ void red_add(double* p, double v) {
    asm volatile("red.relaxed.gpu.global.add.f64 [%0], %1;" ::"l"(p), "d"(v));
}

// C += the warp's 32 x 32 part; LOWER: entries with column <= row + diag only (what lies above
// the diagonal stays as it was)
template <bool LOWER>
__device__ __forceinline__ void add_tile(double* C, int ldc, const double* row_scale, const double* col_scale,
                                         const int (&top)[4][16], const unsigned (&low)[4][16], int gr, int t4, int diag) {
#pragma unroll
    for (int h = 0; h < 4; ++h)
#pragma unroll
        for (int o = 0; o < 2; ++o) {
            const int r = 16 * (h >> 1) + 8 * o + gr;
            double* p = C + (size_t)r * ldc + 2 * t4;
            const double sr = row_scale[r];
#pragma unroll
            for (int j = 0; j < 4; ++j)
#pragma unroll
                for (int z = 0; z < 2; ++z) {
                    const int e = 4 * j + 2 * o + z, c = 32 * (h & 1) + 8 * j + z;
                    const double v = to_double(top[h][e], low[h][e]) * sr * col_scale[c + 2 * t4];
                    if (!LOWER || c + 2 * t4 <= r + diag) red_add(p + c, v);
                }
        }
}

// a tile: its entry (0, 0) in C, its first rows in A and B, in 128s
struct Tile {
    int64_t c;
    int rows, cols;
    bool skip, lower;  // above the diagonal; crosses it
};
__device__ __forceinline__ Tile decode(const SplitArgs& a, int64_t item) {
    const int side = a.bsz >> 7, lg = a.bsz == 256 ? 2 : 0;
    const int64_t p = item >> lg;
    const int e = (int)item & ((1 << lg) - 1), ti = e >> (lg >> 1), tj = e & (side - 1);
    int rr, cc;
    if (a.rows > 0) {
        rr = (int)(p % a.rows);
        cc = (int)(p / a.rows);
    } else {
        grouped_pair(p, a.cols, &rr, &cc);
    }
    const int64_t r = a.r0 + rr, c = a.c0 + cc;
    Tile t;
    t.c = ((a.by_rows ? tri64(r) + c : block_id(r, c, a.nb)) * a.bsz + ti * 128) * a.bsz + tj * 128;
    t.rows = (a.offset + rr) * side + ti;
    t.cols = (a.offset + cc) * side + tj;
    t.skip = a.rows == 0 && t.rows < t.cols;
    t.lower = a.rows == 0 && t.rows == t.cols;
    return t;
}

// One CTA: kPerCta consecutive 128 x 128 tiles, two passes each: levels 7..4 (24 plane
// products, all planes), then 3..0 (10 products of planes 0..3).  A pass's four levels are
// four accumulators of 128 columns, the whole of TMEM; in a pass's last K chunk the levels
// are finished one by one and in the next pass's first chunk begun one by one, so that the
// epilogue warps drain a level while the others are being computed.  C gets one add an
// entry, without a load: a load waits behind the copies' queue (a tile took 24 to 38 us that
// way), and the adds run at the L2's rate for FP64 (12 us a tile, beside the products).
// N = 64 would read shared memory 1.5 times as fast as it delivers.  Pairs of SMs
// (cta_group::2) and stages of half the depth were slower: their smaller copies take
// longer than the products (11 and 10 us a tile against 7.5).
// A tile of a 256-wide panel takes an SM 19.4 us (45 us on the FP64 pipe; 12 without the
// adds); the update of 62 block columns of 256 2.15 -> 1.01 ms.  Two panels at once do twice
// the products for the same adds: the top level's sums then just fit (512 x 127^2 x 256
// < 2^31).
__global__ void __launch_bounds__(kThreads, 1) split_update_kernel(SplitArgs a) {
    extern __shared__ uint8_t raw[];
    uint8_t* smem = reinterpret_cast<uint8_t*>((reinterpret_cast<uintptr_t>(raw) + 511) & ~(uintptr_t)511);
    double* scales = reinterpret_cast<double*>(smem + kStages * kStage);  // 128 rows, 128 columns
    uint64_t* bars = reinterpret_cast<uint64_t*>(scales + 256);
    uint64_t *full = bars, *empty = bars + kStages, *tfull = empty + kStages, *tempty = tfull + 4, *drained = tempty + 4;
    uint32_t* slot = reinterpret_cast<uint32_t*>(drained + 1);
    __shared__ Tile tiles[kPerCta];
    __shared__ Waits s_waits;
    volatile Waits* waits = &s_waits;
    const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
    if (threadIdx.x == 0) {
        for (int i = 0; i < kStages; ++i) {
            mbar_init(&full[i], 1);
            mbar_init(&empty[i], 1);
        }
        for (int i = 0; i < 4; ++i) {
            mbar_init(&tfull[i], 1);
            mbar_init(&tempty[i], kEpi);
        }
        mbar_init(drained, 1);
        s_waits.fail = 0;
        s_waits.limit = kWaitClk;
        fence_barrier_init();
    }
    if (warp == 0) {
        tmem_alloc(slot, 512);
        tmem_relinquish();
    }
    if (warp == 2 && lane < kPerCta && (int64_t)blockIdx.x * kPerCta + lane < a.items)
        tiles[lane] = decode(a, (int64_t)blockIdx.x * kPerCta + lane);
    tc_fence_before();
    __syncthreads();
    tc_fence_after();
    const uint32_t taddr = *slot;
    const int count = (int)min((int64_t)kPerCta, a.items - (int64_t)blockIdx.x * kPerCta);
    const int chunks = a.depth / kKc;

    if (warp == 0) {
        if (lane == 0) {
            uint32_t g = 0;
            bool ok = true;
            for (int it = 0; it < count && ok; ++it) {
                const Tile t = tiles[it];
                if (t.skip) continue;
                const int8_t* dA = a.digA + (int64_t)t.rows * chunks * kOperand;
                const int8_t* dB = a.digB + (int64_t)t.cols * chunks * kOperand;
                for (int pass = 0; pass < 2 && ok; ++pass) {
                    const uint32_t bytes = (pass ? kHighPlanes : kPlanes) * kPlane;
                    for (int kc = 0; kc < chunks; ++kc, ++g) {
                        const uint32_t s = g % kStages;
                        if (g >= kStages && !suspended_wait(&empty[s], (g / kStages - 1) & 1, waits)) {
                            ok = false;
                            break;
                        }
                        uint8_t* st = smem + s * kStage;
                        mbar_arrive_expect_tx(&full[s], 2 * bytes);
                        bulk_load(st, dA + kc * kOperand, bytes, &full[s]);
                        bulk_load(st + kOperand, dB + kc * kOperand, bytes, &full[s]);
                    }
                }
            }
            // no load may still be writing into shared memory when the CTA leaves
            for (uint32_t h = g > kStages ? g - kStages : 0; h < g; ++h) landed(&full[h % kStages], (h / kStages) & 1, waits);
        }
    } else if (warp == 1) {
        const bool leader = elect_one();  // the whole warp walks the loop, so that descriptors stay in uniform registers
        uint32_t g = 0, u = 0;
        bool ok = true;
        for (int it = 0; it < count && ok; ++it) {
            if (tiles[it].skip) continue;
            for (int pass = 0; pass < 2 && ok; ++pass, ++u) {
                for (int kc = 0; kc < chunks; ++kc, ++g) {
                    const uint32_t s = g % kStages;
                    if (!(ok = suspended_wait_warp(&full[s], (g / kStages) & 1, waits))) break;
                    tc_fence_after();
                    const uint64_t da = umma_desc_sw64(smem_u32(smem + s * kStage));
                    uint64_t* wait = kc == 0 && u > 0 ? tempty : nullptr;
                    uint64_t* done = kc == chunks - 1 ? tfull : nullptr;
                    ok = pass == 0 ? issue_levels<kHighPlanes>(taddr, da, kc > 0, wait, done, (u - 1) & 1, leader, waits)
                                   : issue_levels<0>(taddr, da, kc > 0, wait, done, (u - 1) & 1, leader, waits);
                    if (!ok) break;
                    if (leader) umma_commit(&empty[s]);
                    __syncwarp();
                }
            }
        }
        // TMEM is released only after every MMA issued here has completed
        if (leader) umma_commit(drained);
        __syncwarp();
        const long long t0 = clock64();
        while (!mbar_try_wait(drained, 0) && clock64() - t0 < kWaitClk) {}
    } else {
        // warp: rows 32 q .. +31 and 32 columns of the tile.  TMEM is read in 16 x 32 pieces
        // whose lane (g, t) holds rows g and g + 8, columns 8 j + 2 t and the next: an access to
        // C takes 64 bytes of each of eight rows (a row a lane: 32 lines an access).
        const int q = warp & 3, col0 = ((warp - 2) >> 2) * 64, gr = lane >> 2, t4 = lane & 3;
        const uint32_t tcol = taddr + ((uint32_t)(q * 32) << 16) + col0;
        uint32_t u = 0;
        bool ok = true;
        for (int it = 0; it < count; ++it) {  // also after a wait ran out: the barriers below
            const Tile t = tiles[it];
            if (t.skip) continue;
            double* C = a.C + t.c + (int64_t)(32 * q) * a.bsz + col0;
            const int e = threadIdx.x - 64;
            const double sc = e < 128 ? a.sign * a.scaleA[(int64_t)t.rows * 128 + e]
                                      : a.scaleB[(int64_t)t.cols * 128 + e - 128];
            asm volatile("bar.sync 1, 256;" ::: "memory");  // every warp has read the last tile's
            if (e < 256) scales[e] = sc;
            asm volatile("bar.sync 1, 256;" ::: "memory");
            // The levels come lowest first and each is carried into the next, so that 32 bits do:
            // top = the sum so far in the last level's unit, low = the bytes below it (the
            // last one 2^-56; of levels 6 and 7 only the carry, rounded to nearest).
            int top[4][16];  // [row half, column half]
            unsigned low[4][16];
#pragma unroll
            for (int pass = 0; pass < 2; ++pass) {
#pragma unroll
                for (int x = 0; x < 4; ++x) {
                    if (ok) ok = suspended_wait_warp(&tfull[x], (u + pass) & 1, waits);
                    if (!ok) continue;
                    tc_fence_after();
#pragma unroll
                    for (int h = 0; h < 4; ++h) {
                        uint32_t v[16];
                        tmem_ld_16x256b_x4(tcol + ((uint32_t)(16 * (h >> 1)) << 16) + x * 128 + (h & 1) * 32, v);
                        tmem_ld_wait();
#pragma unroll
                        for (int e = 0; e < 16; ++e) {
                            int& w = top[h][e];
                            const int p = (int)v[e], level = pass ? 3 - x : 7 - x;
                            if (level == 4)
                                low[h][e] = (unsigned)w << 24;
                            else if (level < 4 && level > 0)
                                low[h][e] = __funnelshift_r(low[h][e], w, 8);
                            w = level == 7 ? p + (1 << 15) : level > 0 ? (w >> 8) + p : w + p * 256;
                        }
                    }
                    tc_fence_before();
                    __syncwarp();
                    if (lane == 0) mbar_arrive(&tempty[x]);
                }
            }
            if (!ok) continue;
            u += 2;
            if (t.lower)
                add_tile<true>(C, a.bsz, scales + 32 * q, scales + 128 + col0, top, low, gr, t4, 32 * q - col0);
            else
                add_tile<false>(C, a.bsz, scales + 32 * q, scales + 128 + col0, top, low, gr, t4, 0);
        }
    }
    tc_fence_before();
    __syncthreads();
    if (threadIdx.x == 0 && s_waits.fail) atomicMin(a.info, -1ll);
    if (warp == 0) tmem_dealloc(taddr, 512);
}


size_t digits_bytes(int64_t rows, int depth) { return (size_t)rows * (depth * kPlanes + sizeof(double)); }

hs_status launch_products(hs_ctx ctx, SplitArgs& a, cudaStream_t s) {
    const int64_t blocks = a.rows > 0 ? (int64_t)a.rows * a.cols : tri64(a.cols);
    a.nb = ctx->nb;
    a.bsz = ctx->bsz;
    a.items = blocks * (a.bsz / 128) * (a.bsz / 128);
    a.info = ctx->d_info;
    const int64_t grid = (a.items + kPerCta - 1) / kPerCta;
    HS_REQUIRE(grid < (1LL << 31), "too many tiles for one launch");
    HS_CUDA(cudaFuncSetAttribute(split_update_kernel, cudaFuncAttributeMaxDynamicSharedMemorySize, kSmem));
    ctx->launches += 1;
    split_update_kernel<<<(unsigned)grid, kThreads, kSmem, s>>>(a);
    HS_CHECK_LAUNCH("split_update");
    return HS_OK;
}

}  // namespace

size_t split_update_bytes(int nb, int bsz, int panels) { return digits_bytes((int64_t)(nb - panels) * bsz, panels * bsz); }

hs_status launch_split_update(hs_ctx ctx, double* A, int k, int panels, int colStart, void* ws, cudaStream_t s) {
    const int nb = ctx->nb, bsz = ctx->bsz, row0 = k + panels;
    const size_t bb = (size_t)bsz * bsz;
    const int64_t rows = (int64_t)(nb - row0) * bsz;
    SplitArgs a{};
    a.depth = panels * bsz;
    HS_REQUIRE(a.depth == 256 || a.depth == 512, "one or two panels of 256, or two of 128");
    int8_t* D = static_cast<int8_t*>(ws);
    double* scale = reinterpret_cast<double*>(D + rows * a.depth * kPlanes);
    const double* P0 = A + (size_t)block_id(row0, k, nb) * bb;
    const double* P1 = panels == 2 ? A + (size_t)block_id(row0, k + 1, nb) * bb : P0;
    prof_begin(ctx, s, HS_KERNEL_UPDATE);
    ctx->launches += 1;
    if (a.depth == 512)
        digits_kernel<512><<<(unsigned)(rows / 8), 256, 0, s>>>(P0, P1, bsz, rows, D, scale);
    else
        digits_kernel<256><<<(unsigned)(rows / 8), 256, 0, s>>>(P0, P1, bsz, rows, D, scale);
    HS_CHECK_LAUNCH("split_digits");
    a.C = A;
    a.digA = a.digB = D;
    a.scaleA = a.scaleB = scale;
    a.sign = -1.0;
    a.cols = nb - colStart;
    a.r0 = a.c0 = colStart;
    a.offset = colStart - row0;
    hs_status st = launch_products(ctx, a, s);
    if (st != HS_OK) return st;
    const double n = bsz, m = a.cols, blocks = m * (m + 1) / 2;
    prof_end(ctx, s, HS_KERNEL_UPDATE, panels * ((blocks - m) * 2.0 * n * n * n + m * n * n * (n + 1.0)),
             (2.0 * blocks + panels * m) * n * n * 8.0);
    return HS_OK;
}

size_t split_inverse_bytes(int nb) { return 3 * digits_bytes((int64_t)nb * 256, 256); }

hs_status launch_split_inverse_step(hs_ctx ctx, double* L, int k, const double* W, double* S, void* ws,
                                    cudaStream_t s, cudaStream_t side,
                                    cudaEvent_t (&done)[2]) {
    const int nb = ctx->nb;
    const size_t bb = 65536;
    HS_REQUIRE(ctx->bsz == 256, "blocks of 256");
    const int64_t cap = (int64_t)nb * 256;
    const size_t one = digits_bytes(cap, 256);
    int8_t *DW = static_cast<int8_t*>(ws) + (k & 1) * one, *DL = static_cast<int8_t*>(ws) + 2 * one;
    double* scaleW = reinterpret_cast<double*>(DW + cap * 256 * kPlanes);
    double* scaleL = reinterpret_cast<double*>(DL + cap * 256 * kPlanes);
    if (k >= 2) HS_CUDA(cudaStreamWaitEvent(s, done[k & 1], 0));  // step k - 2's product with itself
    prof_begin(ctx, s, HS_KERNEL_ADJOINT);
    ctx->launches += 1;
    digits_transposed_kernel<<<dim3(16, k + 1), 256, 0, s>>>(W, DW, scaleW);
    HS_CHECK_LAUNCH("digits_transposed");
    SplitArgs a{};
    a.depth = 256;
    a.digB = DW;
    a.scaleB = scaleW;
    hs_status st;
    const int below = nb - k - 1;
    if (below > 0) {
        const int64_t rows = (int64_t)below * 256;
        ctx->launches += 1;
        const double* P = L + (size_t)block_id(k + 1, k, nb) * bb;
        digits_kernel<256><<<(unsigned)(rows / 8), 256, 0, s>>>(P, nullptr, 256, rows, DL, scaleL);
        HS_CHECK_LAUNCH("split_digits");
        a.C = S;
        a.by_rows = 1;
        a.digA = DL;
        a.scaleA = scaleL;
        a.sign = -1.0;
        a.rows = below;
        a.cols = k + 1;
        a.r0 = k + 1;
    }
    HS_CUDA(cudaEventRecord(ctx->ev_a, s));
    HS_CUDA(cudaStreamWaitEvent(side, ctx->ev_a, 0));
    if (below > 0 && (st = launch_products(ctx, a, s)) != HS_OK) return st;
    HS_CUDA(cudaMemsetAsync(L + (size_t)block_id(k, k, nb) * bb, 0, (size_t)(nb - k) * bb * sizeof(double), side));
    a.C = L;
    a.by_rows = 0;
    a.digA = DW;
    a.scaleA = scaleW;
    a.sign = 1.0;
    a.rows = 0;
    a.cols = k + 1;
    a.r0 = 0;
    if ((st = launch_products(ctx, a, side)) != HS_OK) return st;
    HS_CUDA(cudaEventRecord(done[k & 1], side));
    const double blocks = (double)below * (k + 1) + 0.5 * (k + 1) * (k + 2), n = 256;
    prof_end(ctx, s, HS_KERNEL_ADJOINT, 2.0 * blocks * n * n * n, 2.0 * blocks * n * n * 8.0);
    return HS_OK;
}

}  // namespace hs
