// k_diag.cu — one diagonal block of the blocked Cholesky in FP64: factor L and inverse
// L^-1 together (the panel TRSM and the triangular sweeps are products with the inverse),
// and the inverses alone of all diagonal blocks of a factor.
//
// Reference kernel replaced: MatrixOperations.cpp:7-191 (cholesky{,_GPU,_optimizedGPU});
// the inverse has no counterpart there.
//
// The block is the serial chain of a factorisation: nothing else of the next column can
// start before it is done, so its latency, not its 4/3 n^3 flops, is what counts.  A
// 128 x 128 block stays in one CTA's shared memory from load to store: L on and below the
// diagonal of a square, Y = L^-T (upper triangular) above it, their 32 x 32 diagonal
// blocks apart.  For each of the four 32-column panels p:
//   F   warp 0 factors the diagonal block (panel_diag) and warp 1 inverts it 8 columns
//       behind (panel_inverse).  Beside them, off their scheduler, eight warps run on the
//       FP64 tensor pipe (m8n8k4): panel p-1's update of the columns after p, and
//       T_Rp = -sum over R <= q < p of Y_Rq L_pq^T, what Y's column p needs of the
//       panels before; other warps load and store.
//   TR  the rows of L below the diagonal block times Y_pp, and Y_Rp = T_Rp Y_pp: always
//       96 rows together, 8 a warp
//   U   the next diagonal block, the one part of the update that F waits for
// A 256 x 256 block is 2 x 2 of such blocks: A11, L21 = A21 L11^-T, A22 -= L21 L21^T,
// A22, and Y12 = -(Y11 L21^T) Y22, the products split over the CTAs of a cluster.
//
// What bounds it: the 64 steps of warp 0 (about 5.5k cycles a panel of the 9k it takes) and
// getting the results out (27 bytes a cycle).  Measured alone, factor and inverse: 128:
// 24.6 us, 256: 65 us with 8 CTAs, 150 us with one; the kernels before it (POTRF in shared
// memory, then the substitution of an identity) took 147 + 114 us for 128 and ~600 us for
// 256, and the mixed factor's one-CTA kernel that kept the block in L2 86 and 200 us.
#include "hs_internal.cuh"

namespace hs {
namespace {

constexpr int kN = 128;          // on-chip block
constexpr int kThreads = 384;     // 12 warps, up to 168 registers a thread: a row of 32 doubles stays in registers
constexpr int kLdS = 132;         // square: rows 32 bytes apart modulo 128, so that a fragment's 4 rows x 4
                                  // columns of doubles are a conflict-free phase
constexpr int kLdY = 36;          // the diagonal blocks of Y likewise
constexpr size_t kSmemBytes = (size_t)(kN * kLdS + 4 * 32 * kLdY + kN) * sizeof(double);

struct DiagArgs {
    const double* in64;   // the block (row major), or
    const float* in32;    // the same in FP32 (in64 null)
    double* L;            // factor out (may be in64); null with FACTOR false
    int pad_sqrt;         // L is in place: padding rows untouched but for sqrt of their diagonal entry, and
                          // zeros above the diagonal inside the 32 x 32 diagonal blocks
    int write_upper;      // L: the other zeros above the diagonal too
    double* Y;            // L^-T row major (null: not written; bsz 256 then keeps that of the first 128 rows in
                          // L's upper right quadrant until the zeros go there)
    int y_full;           // Y: all of its zeros (the inverses alone); else only those beside its 64 x 64 diagonal blocks
    double* T;            // bsz 256: a 128 x 128 scratch block
    float *invHi, *invLo; // L^-1 in FP32 and its low part under TF32 truncation (null: not written)
    int zero_upper;       // invHi / invLo: also write the part above the diagonal
    int valid;            // rows / columns from here on are padding (identity in the inverse)
    long long* info;      // [0] smallest failing pivot row, [1] most negative failing pivot (if record_neg)
    int record_neg;
    long long row_base;
    int ld;               // leading dimension of every array: bsz
    // batched inverses (FACTOR false): block k of the packed factor at `in64`, Y block k
    int nb;
    int64_t N;
};

// the shared arrays, taken from the extern array at every use so that the address space is
// known wherever a function is not inlined
struct Smem {
    struct S_ {  // the square
        __device__ __forceinline__ operator double*() const;
    } S;
    struct Yd_ {  // [p][row][column]: diagonal block p of Y, zero below its diagonal
        __device__ __forceinline__ operator double*() const;
    } Yd;
    struct ri_ {  // reciprocal diagonal of L
        __device__ __forceinline__ operator double*() const;
    } ri;
};
extern __shared__ __align__(16) double diag_smem[];
__device__ __forceinline__ Smem::S_::operator double*() const { return diag_smem; }
__device__ __forceinline__ Smem::Yd_::operator double*() const { return diag_smem + kN * kLdS; }
__device__ __forceinline__ Smem::ri_::operator double*() const { return diag_smem + kN * kLdS + 4 * 32 * kLdY; }
__device__ __forceinline__ void bar_sync(int id, int count) {
    asm volatile("bar.sync %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void bar_arrive(int id, int count) {
    asm volatile("bar.arrive %0, %1;" ::"r"(id), "r"(count) : "memory");
}
__device__ __forceinline__ void cluster_sync() {
    asm volatile("barrier.cluster.arrive.release.aligned;\n\tbarrier.cluster.wait.acquire.aligned;" ::: "memory");
}
__device__ __forceinline__ unsigned cluster_rank() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_ctarank;" : "=r"(r));
    return r;
}
__device__ __forceinline__ unsigned cluster_size() {
    unsigned r;
    asm volatile("mov.u32 %0, %%cluster_nctarank;" : "=r"(r));
    return r;
}

// 1 / sqrt(a) for a in the normal range, without a branch: the hardware's approximation
// and one step of Householder's third-order iteration, y (1 + e/2 + 3/8 e^2) with
// e = 1 - a y^2 (the Taylor series of (1 - e)^-1/2)
__device__ __forceinline__ double rsqrt_step(double a) {
    double y;
    asm("rsqrt.approx.ftz.f64 %0, %1;" : "=d"(y) : "d"(a));
    const double e = fma(-(a * y), y, 1.0);
    return fma(y * e, fma(0.375, e, 0.5), y);
}

// p in [2^-465, 2^465), det in [2^-963, inf), by their high words (off the FP64 pipe)
__device__ __forceinline__ bool pivot_safe(double p) {
    return (unsigned)(__double2hiint(p) - 0x22E00000) < 0x5D000000u - 0x22E00000u;
}
__device__ __forceinline__ bool det_safe(double d) {
    return (unsigned)(__double2hiint(d) - 0x03C00000) < 0x7FF00000u - 0x03C00000u;
}

// 8 columns of the panel's diagonal block for any input, one after the other (lane = row):
// x in and out, reciprocal diagonal into ri; records failing pivots
__device__ __noinline__ void sub_panel_general(double (&x)[8], double* ri, int s, int lane, long long* info,
                                               int record_neg, long long row, int n_valid) {
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const int kk = 8 * s + k;
        const double p = __shfl_sync(0xffffffffu, x[k], kk);
        if (lane == 0 && !(p > 0.0) && k < n_valid) {
            atomicMin(info, row + k);
            // a larger signed pattern is a larger magnitude; NaN and zero pivots are not recorded
            if (record_neg && p < 0.0) atomicMax(info + 1, __double_as_longlong(p));
        }
        const double r = rsqrt(p);
        const double l = lane == kk ? sqrt(p) : (lane > kk ? x[k] * r : 0.0);
        x[k] = l;
        if (lane == 0) ri[kk] = r;
#pragma unroll
        for (int j = k + 1; j < 8; ++j) x[j] = fma(-l, __shfl_sync(0xffffffffu, l, 8 * s + j), x[j]);
    }
}

// the 8 x 8 tiles (rt, ct), S < ct <= rt, of the panel's diagonal block after its columns
// 8 S .. 8 S + 7, all in flight together, one warp
template <int S>
__device__ __forceinline__ void diag_trailing(const Smem m, int c0, int g, int t) {
    constexpr int kT = (3 - S) * (4 - S) / 2;
    double acc[kT][2], ar[4][2];
#pragma unroll
    for (int i = S + 1; i < 4; ++i) {
        const double* pr = m.S + (c0 + 8 * i + g) * kLdS + c0 + 8 * S + t;
        ar[i][0] = pr[0];
        ar[i][1] = pr[4];
    }
    int u = 0;
#pragma unroll
    for (int ct = S + 1; ct < 4; ++ct)
#pragma unroll
        for (int rt = ct; rt < 4; ++rt, ++u) {
            acc[u][0] = acc[u][1] = 0.0;
            dmma884(acc[u], ar[rt][0], ar[ct][0]);
            dmma884(acc[u], ar[rt][1], ar[ct][1]);
        }
    u = 0;
#pragma unroll
    for (int ct = S + 1; ct < 4; ++ct)
#pragma unroll
        for (int rt = ct; rt < 4; ++rt, ++u) {
            double2* q = reinterpret_cast<double2*>(m.S + (c0 + 8 * rt + g) * kLdS + c0 + 8 * ct + 2 * t);
            const double2 v = *q;
            *q = make_double2(v.x - acc[u][0], v.y - acc[u][1]);
        }
}

// warp 0: L of the panel's diagonal block (rows / columns c0 ..), its reciprocal diagonal
// in ri; warp 1 is released after every 8 columns.  Every lane
// factors the 8 x 8 block on the diagonal in its own registers, two columns a step, with
// no exchange between the lanes in the chain of pivots (with a shuffle and a broadcast
// through shared memory a step instead: 424 cycles a step), then solves its own row of
// the 8 columns.  The rest of the block is brought up to date by two DMMAs a tile.  The
// steps are free of branches: a pivot outside the range their product form is safe in
// sends the 8 columns through sub_panel_general instead.
__device__ __forceinline__ void panel_diag(const Smem m, int c0, int lane, const DiagArgs& a, int d0) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
        const int cs = c0 + 8 * s;
        double x[8];
        double* row = m.S + (c0 + lane) * kLdS + cs;
        auto load = [&]() {
#pragma unroll
            for (int j = 0; j < 8; j += 2) {
                const double2 v = *reinterpret_cast<const double2*>(row + j);
                x[j] = 8 * s + j <= lane ? v.x : 0.0;
                x[j + 1] = 8 * s + j + 1 <= lane ? v.y : 0.0;
            }
        };
        double d[8][8];
#pragma unroll
        for (int i = 0; i < 8; ++i)
#pragma unroll
            for (int j = 0; j <= i; j += 2) {
                const double2 v = *reinterpret_cast<const double2*>(m.S + (cs + i) * kLdS + cs + j);
                d[i][j] = v.x;
                if (j + 1 <= i) d[i][j + 1] = v.y;
            }
        load();
        bool safe = true;
        double ri[8];
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
            const double p = d[k][k], b = d[k + 1][k], c = d[k + 1][k + 1];
            const double det = fma(p, c, -(b * b));
            // p c must neither overflow nor lose its low bits
            safe = safe && pivot_safe(p) && pivot_safe(c) && det_safe(det);
            const double r1 = rsqrt_step(p), rd = rsqrt_step(det);
            const double l11 = p * r1, l21 = b * r1, r2 = rd * l11;
            ri[k] = r1;
            ri[k + 1] = r2;
            d[k][k] = l11;
            d[k + 1][k] = l21;
            d[k + 1][k + 1] = (det * rd) * r1;
#pragma unroll
            for (int i = k + 2; i < 8; ++i) {
                d[i][k] *= r1;
                d[i][k + 1] = fma(-d[i][k], l21, d[i][k + 1]) * r2;
            }
#pragma unroll
            for (int i = k + 2; i < 8; ++i)
#pragma unroll
                for (int j = k + 2; j <= i; ++j) {
                    d[i][j] = fma(-d[i][k], d[j][k], d[i][j]);
                    d[i][j] = fma(-d[i][k + 1], d[j][k + 1], d[i][j]);
                }
        }
        // this lane's row against it: a row below it is a substitution, and a row of the
        // block itself comes out as its row of L (what lies above the diagonal is not read)
#pragma unroll
        for (int k = 0; k < 8; ++k) {
            x[k] *= ri[k];
#pragma unroll
            for (int j = k + 1; j < 8; ++j) x[j] = fma(-x[k], d[j][k], x[j]);
        }
        if (lane == 0) {
#pragma unroll
            for (int k = 0; k < 8; k += 2) *reinterpret_cast<double2*>(m.ri + cs + k) = make_double2(ri[k], ri[k + 1]);
        }
        if (!safe) {  // the same for every lane
            load();
            double w[8];  // a copy of its own: x stays in registers
#pragma unroll
            for (int j = 0; j < 8; ++j) w[j] = x[j];
            sub_panel_general(w, m.ri + c0, s, lane, a.info, a.record_neg, a.row_base + d0 + 8 * s, a.valid - d0 - 8 * s);
#pragma unroll
            for (int j = 0; j < 8; ++j) x[j] = w[j];
        }
#pragma unroll
        for (int j = 0; j < 8; ++j)
            if (8 * s + j <= lane) row[j] = x[j];
        __syncwarp();
        bar_arrive(1 + s, 64);
        if (s == 0)
            diag_trailing<0>(m, c0, g, t);
        else if (s == 1)
            diag_trailing<1>(m, c0, g, t);
        else if (s == 2)
            diag_trailing<2>(m, c0, g, t);
        __syncwarp();
    }
}

// one warp: Y_pp = L_pp^-T of diagonal block p into Yd, by substitution of the identity's
// rows (lane = row), 8 columns at a time: behind warp 0 (FACTOR) or from a given factor
template <bool FACTOR>
__device__ __forceinline__ void panel_inverse(const Smem m, int p, int lane) {
    const int c0 = 32 * p, g = lane >> 2, t = lane & 3;
    double* Y = m.Yd + p * 32 * kLdY;
    if (!FACTOR) {
        m.ri[c0 + lane] = 1.0 / m.S[(c0 + lane) * kLdS + c0 + lane];
        __syncwarp();
    }
#pragma unroll 1
    for (int s = 0; s < 4; ++s) {
        const int cs = c0 + 8 * s;
        const int st = s - lane / 8;  // > 0: under way, 0: the row starts here, < 0: still zero
        double x[8];
        double* row = Y + lane * kLdY + 8 * s;
#pragma unroll
        for (int j = 0; j < 8; j += 2) {
            const double2 v = *reinterpret_cast<const double2*>(row + j);
            x[j] = st > 0 ? v.x : (st == 0 && j == lane % 8 ? 1.0 : 0.0);
            x[j + 1] = st > 0 ? v.y : (st == 0 && j + 1 == lane % 8 ? 1.0 : 0.0);
        }
        if (FACTOR) bar_sync(1 + s, 64);
        const double* L = m.S + cs * kLdS + cs;
#pragma unroll
        for (int k = 0; k < 8; k += 2) {
            const double2 rr = *reinterpret_cast<const double2*>(m.ri + cs + k);
            const double p0 = x[k] * rr.x;
            const double p1 = fma(-p0, L[(k + 1) * kLdS + k], x[k + 1]) * rr.y;
            x[k] = p0;
            x[k + 1] = p1;
#pragma unroll
            for (int j = k + 2; j < 8; ++j) {
                const double2 l = *reinterpret_cast<const double2*>(L + j * kLdS + k);
                x[j] = fma(-p0, l.x, x[j]);
                x[j] = fma(-p1, l.y, x[j]);
            }
        }
#pragma unroll
        for (int j = 0; j < 8; j += 2) *reinterpret_cast<double2*>(row + j) = make_double2(x[j], x[j + 1]);
        __syncwarp();
#pragma unroll 1
        for (int ct = s + 1; ct < 4; ++ct) {
            const double* pb = m.S + (c0 + 8 * ct + g) * kLdS + cs + t;
            const double b0 = pb[0], b1 = pb[4];
#pragma unroll
            for (int rt = 0; rt < 3; ++rt)
                if (rt <= s) {
                    const double* pa = Y + (8 * rt + g) * kLdY + 8 * s + t;
                    double acc[2] = {0.0, 0.0};
                    dmma884(acc, pa[0], b0);
                    dmma884(acc, pa[4], b1);
                    double2* q = reinterpret_cast<double2*>(Y + (8 * rt + g) * kLdY + 8 * ct + 2 * t);
                    const double2 v = rt == s ? make_double2(0.0, 0.0) : *q;
                    *q = make_double2(v.x - acc[0], v.y - acc[1]);
                }
        }
        __syncwarp();
    }
}

// one warp: acc (8 rows, the first `nt` tiles of 8 columns) += A B^T over 32 columns, A's
// fragment row at pa, B's at pb (row major)
__device__ __forceinline__ void strip_nt(double (&acc)[4][2], const double* pa, const double* pb, int nt = 4) {
#pragma unroll
    for (int k0 = 0; k0 < 32; k0 += 4) {
        const double av = pa[k0];
#pragma unroll
        for (int ni = 0; ni < 4; ++ni)
            if (ni < nt) dmma884(acc[ni], av, pb[8 * ni * kLdS + k0]);
    }
}

// rows 8 sub .. of the 32 x 32 tile (R, C) of A, its first `nt` 8-column tiles:
// S -= L_Rp L_Cp^T
__device__ __forceinline__ void update_strip(const Smem m, int p, int R, int C, int sub, int nt, int lane) {
    const int g = lane >> 2, t = lane & 3, r = 32 * R + 8 * sub + g;
    double acc[4][2] = {};
    strip_nt(acc, m.S + r * kLdS + 32 * p + t, m.S + (32 * C + g) * kLdS + 32 * p + t, nt);
#pragma unroll
    for (int ni = 0; ni < 4; ++ni) {
        if (ni >= nt) break;
        double2* q = reinterpret_cast<double2*>(m.S + r * kLdS + 32 * C + 8 * ni + 2 * t);
        const double2 v = *q;
        *q = make_double2(v.x - acc[ni][0], v.y - acc[ni][1]);
    }
}

// rows 8 sub .. of T_Rp = -sum over R <= q < p of Y_Rq L_pq^T, into the square above the
// diagonal
__device__ __forceinline__ void inverse_strip(const Smem m, int p, int R, int sub, int lane) {
    const int g = lane >> 2, t = lane & 3, r = 32 * R + 8 * sub + g;
    double acc[4][2] = {};
    const double* pb = m.S + (32 * p + g) * kLdS + t;
    strip_nt(acc, m.Yd + (32 * R + 8 * sub + g) * kLdY + t, pb + 32 * R);
#pragma unroll 1
    for (int q = R + 1; q < p; ++q) strip_nt(acc, m.S + r * kLdS + 32 * q + t, pb + 32 * q);
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
        *reinterpret_cast<double2*>(m.S + r * kLdS + 32 * p + 8 * ni + 2 * t) = make_double2(-acc[ni][0], -acc[ni][1]);
}

// 8 rows of column block p, in place: times Y_pp (upper triangular)
__device__ __forceinline__ void solve_strip(const Smem m, int p, int r0, int lane) {
    const int g = lane >> 2, t = lane & 3;
    double* row = m.S + (r0 + g) * kLdS + 32 * p;
    const double* pb = m.Yd + (32 * p + t) * kLdY + g;
    double acc[4][2] = {};
#pragma unroll
    for (int k0 = 0; k0 < 32; k0 += 4) {
        const double av = row[k0 + t];
#pragma unroll
        for (int ni = k0 / 8; ni < 4; ++ni) dmma884(acc[ni], av, pb[k0 * kLdY + 8 * ni]);
    }
    __syncwarp();
#pragma unroll
    for (int ni = 0; ni < 4; ++ni)
        *reinterpret_cast<double2*>(row + 8 * ni + 2 * t) = make_double2(acc[ni][0], acc[ni][1]);
}

// a 128 x 128 quadrant: where it comes from and goes to
struct Quad {
    const double* in64;  // read through L2: another CTA of the cluster may have written it
    const float* in32;
    double *L, *Y;
    float *invHi, *invLo;
    int ld, valid;  // rows / columns from `valid` on: identity
    int write_upper, pad_sqrt, zero_upper, y_full;
    int d0;  // its first row within the diagonal block
};

// 32 x 32 tile (R, C) of the quadrant into the square, threads t0, t0 + nt, ..
__device__ __forceinline__ void load_tile(const Smem m, const Quad q, int R, int C, int t0, int nt) {
#pragma unroll 2
    for (int e = t0; e < 512; e += nt) {
        const int i = 32 * R + e / 16, j = 32 * C + 2 * (e % 16);
        const size_t o = (size_t)i * q.ld + j;
        double2 v;
        if (q.in64) {
            v = __ldcg(reinterpret_cast<const double2*>(q.in64 + o));
        } else {
            const float2 f = *reinterpret_cast<const float2*>(q.in32 + o);
            v = make_double2(f.x, f.y);
        }
        if (i >= q.valid || j >= q.valid) v.x = i == j ? 1.0 : 0.0;
        if (i >= q.valid || j + 1 >= q.valid) v.y = i == j + 1 ? 1.0 : 0.0;
        *reinterpret_cast<double2*>(m.S + i * kLdS + j) = v;
    }
}

__device__ __forceinline__ float tf32_low(float x) {
    return x - __uint_as_float(__float_as_uint(x) & 0xFFFFE000u);
}

// Stores.  A warp gets a store out every 150 to 350 cycles and all warps together ~27
// bytes a cycle (rows of 256 bytes through the copy engine were no faster), so zeros that
// nothing reads are not written, two warps write a part while the next panel is factored
// and all warps the rest at the end.

// steps [s0, s1) of the finished columns 32 p .. of L, then of Y, two rows a step, by warps
// w0, w0 + nw, ..
constexpr int kEarlySteps = 32;  // a panel's steps that are stored while the next is factored
__device__ __forceinline__ void store_panel(const Smem m, const Quad q, int p, int s0, int s1, int w0, int nw, int lane) {
    const int c0 = 32 * p;
    const int hi = lane >> 4, j = c0 + 2 * (lane & 15);  // 16 pairs of columns a row
    const int l0 = q.write_upper ? 0 : c0 / 2, nl = q.L ? kN / 2 - l0 : 0;
    if (q.Y) s1 = min(s1, nl + (q.y_full ? kN : ((p & 1) ? c0 + 32 : c0 + 64)) / 2);
    else s1 = min(s1, nl);
    for (int u0 = s0 + w0; u0 < s1; u0 += 4 * nw) {
        double2 v[4];
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int u = min(u0 + h * nw, s1 - 1);
            // block row of Y: above p in the square, p in Yd, below zero
            const int i = 2 * (u < nl ? u + l0 : u - nl) + hi;
            v[h] = make_double2(0.0, 0.0);
            if (u < nl || i < c0)
                v[h] = *reinterpret_cast<const double2*>(m.S + i * kLdS + j);
            else if (i < c0 + 32)
                v[h] = *reinterpret_cast<const double2*>(m.Yd + i * kLdY + (j - c0));
        }
#pragma unroll
        for (int h = 0; h < 4; ++h) {
            const int u = u0 + h * nw;
            if (u >= s1) break;
            if (u >= nl) {
                *reinterpret_cast<double2*>(q.Y + (size_t)(2 * (u - nl) + hi) * q.ld + j) = v[h];
                continue;
            }
            const int i = 2 * (u + l0) + hi;
            double* o = q.L + (size_t)i * q.ld + j;
            if (q.pad_sqrt && i >= q.valid) {
                if ((i & ~1) == j) o[i & 1] = sqrt(o[i & 1]);
            } else if (j + 1 <= i) {
                *reinterpret_cast<double2*>(o) = v[h];
            } else if (q.pad_sqrt && i >= c0) {  // in place: zeros above the diagonal of the 32 x 32 block
                *reinterpret_cast<double2*>(o) = make_double2(j <= i ? v[h].x : 0.0, 0.0);
            } else if (q.write_upper) {
                *reinterpret_cast<double2*>(o) = make_double2(0.0, 0.0);
            } else if (j <= i) {
                o[0] = v[h].x;
            }
        }
    }
}

// rows 32 p .. of L^-1 in FP32, 8 rows x 16 columns a step
__device__ __forceinline__ void store_f32(const Smem m, const Quad q, int p, int w0, int nw, int lane) {
    if (!q.invHi) return;
    const int c0 = 32 * p, cols = q.zero_upper ? kN / 16 : (c0 + 32) / 16;
    for (int u = w0; u < 4 * cols; u += nw) {
        const int i = c0 + 8 * (u / cols) + (lane & 7), jj = 16 * (u % cols) + 4 * (lane >> 3);
        float f[4] = {0.f, 0.f, 0.f, 0.f};
        if (jj < c0 + 32) {
#pragma unroll
            for (int e = 0; e < 4; ++e)
                f[e] = (float)(jj < c0 ? m.S[(jj + e) * kLdS + i] : m.Yd[(jj + e) * kLdY + (i - c0)]);
        }
        const size_t o = (size_t)i * q.ld + jj;
        *reinterpret_cast<float4*>(q.invHi + o) = make_float4(f[0], f[1], f[2], f[3]);
        *reinterpret_cast<float4*>(q.invLo + o) = make_float4(tf32_low(f[0]), tf32_low(f[1]), tf32_low(f[2]), tf32_low(f[3]));
    }
}

// L (FACTOR) and Y of one quadrant, from memory to memory
template <bool FACTOR>
__device__ void chain128(const Smem m, const DiagArgs& a, const Quad q) {
    const int tid = threadIdx.x, warp = tid >> 5, lane = tid & 31;
    // 2, 3, 5, 6, 7, 9, 10, 11 -> 0..7; warps 4 and 8 share warp 0's scheduler and only
    // load and store while it factors
    const bool worker = warp > 1 && (warp & 3) != 0;
    const int wk = warp - 2 - (warp > 4) - (warp > 8);
    if (FACTOR) {
        for (int R = 0; R < 4; ++R) load_tile(m, q, R, 0, tid, kThreads);
    } else {
        for (int C = 0; C < 4; ++C)
            for (int R = C; R < 4; ++R) load_tile(m, q, R, C, tid, kThreads);
    }
    __syncthreads();
    if (!FACTOR) {
        if (warp < 4) panel_inverse<false>(m, warp, lane);
        __syncthreads();
    }
#pragma unroll 1
    for (int p = 0; p < 4; ++p) {
        if (FACTOR && warp == 0) {
            panel_diag(m, 32 * p, lane, a, q.d0 + 32 * p);
        } else if (FACTOR && warp == 1) {
            panel_inverse<true>(m, p, lane);
        } else if (FACTOR && p == 0) {
            for (int C = 1; C < 4; ++C)
                for (int R = C; R < 4; ++R) load_tile(m, q, R, C, tid - 64, kThreads - 64);
        } else if (worker && p > 0) {
            // T_Rp of Y, and panel p-1's update of the tiles of A from column p on but its
            // diagonal block's, 2 to 3 strips' work a warp
            const int sub = wk & 3;
            if (wk < 4) {
                inverse_strip(m, p, 0, sub, lane);
                if (FACTOR && p == 1) update_strip(m, 0, 2, 1, sub, 4, lane);
                if (FACTOR && p < 3) update_strip(m, p - 1, p + 1, p + 1, sub, sub + 1, lane);
            } else {
                if (p > 1) inverse_strip(m, p, 1, sub, lane);
                if (p > 2) inverse_strip(m, p, 2, sub, lane);
                if (FACTOR && p < 3) update_strip(m, p - 1, 3, p, sub, 4, lane);
                if (FACTOR && p == 1) {
                    update_strip(m, 0, 3, 2, sub, 4, lane);
                    update_strip(m, 0, 3, 3, sub, sub + 1, lane);
                }
            }
        }
        if (p > 0 && (warp == 4 || warp == 8)) {
            if (q.invHi)
                store_f32(m, q, p - 1, (warp >> 2) - 1, 2, lane);
            else
                store_panel(m, q, p - 1, 0, kEarlySteps, (warp >> 2) - 1, 2, lane);
        }
        __syncthreads();
        // 12 strips: the rows of Y above block row p, the rows of L below
        {
            const int blk = warp >> 2, R = blk < p ? blk : blk + 1;
            if (R < p || FACTOR) solve_strip(m, p, 32 * R + 8 * (warp & 3), lane);
        }
        __syncthreads();
        if (p == 3) break;
        if (FACTOR) {
            // one 8 x 8 tile of the next diagonal block's lower part on each of warps 0..9
            if (warp < 10) {
                const int rt = warp < 1 ? 0 : warp < 3 ? 1 : warp < 6 ? 2 : 3, ct = warp - rt * (rt + 1) / 2;
                const int g = lane >> 2, t = lane & 3, c1 = 32 * (p + 1);
                const double* pa = m.S + (c1 + 8 * rt + g) * kLdS + 32 * p + t;
                const double* pb = m.S + (c1 + 8 * ct + g) * kLdS + 32 * p + t;
                double2* sq = reinterpret_cast<double2*>(m.S + (c1 + 8 * rt + g) * kLdS + c1 + 8 * ct + 2 * t);
                const double2 v = *sq;
                double acc[2][2] = {};
#pragma unroll
                for (int k0 = 0; k0 < 32; k0 += 4) dmma884(acc[(k0 >> 2) & 1], pa[k0], pb[k0]);
                *sq = make_double2(v.x - (acc[0][0] + acc[1][0]), v.y - (acc[0][1] + acc[1][1]));
            }
            __syncthreads();
        }
    }
    for (int p = 0; p < 4; ++p) store_panel(m, q, p, p < 3 && !q.invHi ? kEarlySteps : 0, kN, warp, kThreads / 32, lane);
    store_f32(m, q, 3, warp, kThreads / 32, lane);
}

// quadrant `off` of a block's arrays
__device__ __forceinline__ Quad quadrant(const DiagArgs& a, const double* in64, const float* in32, double* L, double* Y,
                                         int off, int valid) {
    const size_t o = (size_t)off * a.ld + off;
    Quad q;
    q.in64 = in64 ? in64 + o : nullptr;
    q.in32 = in32 ? in32 + o : nullptr;
    q.L = L ? L + o : nullptr;
    q.Y = Y ? Y + o : nullptr;
    q.invHi = a.invHi ? a.invHi + o : nullptr;
    q.invLo = a.invLo ? a.invLo + o : nullptr;
    q.ld = a.ld;
    q.valid = valid;
    q.write_upper = a.write_upper;
    q.pad_sqrt = a.pad_sqrt;
    q.zero_upper = a.zero_upper;
    q.y_full = a.y_full;
    q.d0 = off;
    return q;
}

// one warp: D (8 MT rows x 8 columns) = sum over k in [k0, k1) of A[i][k] B[j][k], both row
// major with leading dimensions lda / ldb, read through L2; k0 and k1 multiples of 8 (a
// step takes 8 values of k in the order 0 2 4 6, 1 3 5 7: both operands alike)
template <int MT>
__device__ __forceinline__ void gemm_nt(const double* __restrict__ A, int lda, const double* __restrict__ B, int ldb,
                                        int k0, int k1, int lane, double (&acc)[MT][2]) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mi = 0; mi < MT; ++mi) acc[mi][0] = acc[mi][1] = 0.0;
    const double* pb = B + (size_t)g * ldb + 2 * t;
    const double* pa = A + (size_t)g * lda + 2 * t;
#pragma unroll 4
    for (int k = k0; k < k1; k += 8) {
        const double2 b = __ldcg(reinterpret_cast<const double2*>(pb + k));
        double2 av[MT];
#pragma unroll
        for (int mi = 0; mi < MT; ++mi) av[mi] = __ldcg(reinterpret_cast<const double2*>(pa + (size_t)8 * mi * lda + k));
#pragma unroll
        for (int mi = 0; mi < MT; ++mi) {
            dmma884(acc[mi], av[mi].x, b.x);
            dmma884(acc[mi], av[mi].y, b.y);
        }
    }
}

// the same with B's rows k: D = sum over k of A[i][k] B[k][j]
template <int MT>
__device__ __forceinline__ void gemm_nn(const double* A, int lda, const double* __restrict__ B, int ldb, int k0, int k1,
                                        int lane, double (&acc)[MT][2]) {
    const int g = lane >> 2, t = lane & 3;
#pragma unroll
    for (int mi = 0; mi < MT; ++mi) acc[mi][0] = acc[mi][1] = 0.0;
    const double* pb = B + (size_t)2 * t * ldb + g;
    const double* pa = A + (size_t)g * lda + 2 * t;
#pragma unroll 4
    for (int k = k0; k < k1; k += 8) {
        const double b0 = __ldcg(pb + (size_t)k * ldb), b1 = __ldcg(pb + (size_t)(k + 1) * ldb);
        double2 av[MT];
#pragma unroll
        for (int mi = 0; mi < MT; ++mi) av[mi] = __ldcg(reinterpret_cast<const double2*>(pa + (size_t)8 * mi * lda + k));
#pragma unroll
        for (int mi = 0; mi < MT; ++mi) {
            dmma884(acc[mi], av[mi].x, b0);
            dmma884(acc[mi], av[mi].y, b1);
        }
    }
}

// the 16 groups of 8 columns over the 12 warps: group g costs `rising` g + 1 or 16 - g
// steps, and the four cheapest share a warp with the next four
template <class F>
__device__ __forceinline__ void for_groups(int warp, bool rising, F f) {
    f(rising ? 15 - warp : warp);
    if (warp >= 8) f(rising ? warp - 8 : warp + 4);
}

// Y12 = -(Y11 L21^T) Y22 in two halves (a cluster barrier between them): strips of 16 rows
// first, first + step, ..; rows of L21 from valid2 on count as zero
constexpr int kMT = 2, kStrip = 8 * kMT, kStrips = kN / kStrip;
__device__ __forceinline__ void inverse_corner_t(const double* Y, const double* L21, double* T, int ld, int valid2,
                                                 int first, int step, int warp, int lane) {
    const int g = lane >> 2, t = lane & 3;
    double acc[kMT][2];
    for (int st = first; st < kStrips; st += step) {
        const int j0 = st * kStrip;
        for_groups(warp, false, [&](int cg) {
            gemm_nt<kMT>(Y + (size_t)j0 * ld, ld, L21 + (size_t)(8 * cg) * ld, ld, j0, kN, lane, acc);
#pragma unroll
            for (int mi = 0; mi < kMT; ++mi) {
                const int i = 8 * cg + 2 * t;
                __stcg(reinterpret_cast<double2*>(T + (size_t)(j0 + 8 * mi + g) * kN + i),
                       make_double2(i < valid2 ? acc[mi][0] : 0.0, i + 1 < valid2 ? acc[mi][1] : 0.0));
            }
        });
    }
}
template <class F>
__device__ __forceinline__ void inverse_corner_y(double* Y, const double* T, int ld, int y_full, int first, int step,
                                                 int warp, int lane, F also) {
    const int g = lane >> 2, t = lane & 3;
    double acc[kMT][2];
    for (int st = first; st < kStrips; st += step) {
        const int j0 = st * kStrip;
        for_groups(warp, true, [&](int cg) {
            gemm_nn<kMT>(T + (size_t)j0 * kN, kN, Y + (size_t)kN * ld + kN + 8 * cg, ld, 0, 8 * (cg + 1), lane, acc);
#pragma unroll
            for (int mi = 0; mi < kMT; ++mi) {
                const int j = j0 + 8 * mi + g, i = 8 * cg + 2 * t;
                const double2 v = make_double2(-acc[mi][0], -acc[mi][1]);
                *reinterpret_cast<double2*>(Y + (size_t)j * ld + kN + i) = v;
                if (y_full) *reinterpret_cast<double2*>(Y + (size_t)(kN + j) * ld + i) = make_double2(0.0, 0.0);
                also(j, i, v);
            }
        });
    }
}

template <int BSZ>
__global__ void __launch_bounds__(kThreads, 1) diag_factor_kernel(DiagArgs a) {
    const Smem m{};
    const unsigned rank = BSZ == 128 ? 0 : cluster_rank();
    // rows of the upper right quadrant are padding only if L21 has none but padding
    double* Y11 = BSZ == 128 || a.Y ? a.Y : (a.valid > kN ? a.L + kN : nullptr);
    if (rank == 0) chain128<true>(m, a, quadrant(a, a.in64, a.in32, a.L, Y11, 0, min(a.valid, kN)));
    if constexpr (BSZ == 256) {
        constexpr int ld = 256, MT = kMT;
        const unsigned nranks = cluster_size();
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31, g = lane >> 2, t = lane & 3;
        const int valid2 = a.valid > kN ? a.valid - kN : 0;
        double* L21 = a.L + (size_t)kN * ld;
        double* L22 = L21 + kN;
        double acc[MT][2];
        cluster_sync();
        // L21 = A21 Y11, strip by strip of rows through shared memory (in place); Y11 is
        // upper triangular: columns 8 cg .. need k < 8 (cg + 1)
        for (int st = rank; st < (Y11 ? kStrips : 0); st += nranks) {
            const int i0 = st * kStrip;
            double* F = m.S;  // the chain is done with it
            __syncthreads();
            for (int e = threadIdx.x; e < kStrip * kN; e += kThreads) {
                const size_t o = (size_t)(kN + i0 + e / kN) * ld + e % kN;
                F[(e / kN) * kLdS + e % kN] =
                    a.in64 ? __ldcg(a.in64 + o) : (i0 + e / kN < valid2 ? (double)a.in32[o] : 0.0);
            }
            __syncthreads();
            for_groups(warp, true, [&](int cg) {
                const double* pb = Y11 + (size_t)2 * t * ld + 8 * cg + g;
#pragma unroll
                for (int mi = 0; mi < MT; ++mi) acc[mi][0] = acc[mi][1] = 0.0;
#pragma unroll 4
                for (int k = 0; k < 8 * (cg + 1); k += 8) {
                    const double b0 = __ldcg(pb + (size_t)k * ld), b1 = __ldcg(pb + (size_t)(k + 1) * ld);
#pragma unroll
                    for (int mi = 0; mi < MT; ++mi) {
                        const double2 v = *reinterpret_cast<const double2*>(F + (8 * mi + g) * kLdS + k + 2 * t);
                        dmma884(acc[mi], v.x, b0);
                        dmma884(acc[mi], v.y, b1);
                    }
                }
#pragma unroll
                for (int mi = 0; mi < MT; ++mi) {
                    const int i = i0 + 8 * mi + g;
                    if (i < valid2 || !a.pad_sqrt)
                        __stcg(reinterpret_cast<double2*>(L21 + (size_t)i * ld + 8 * cg + 2 * t),
                               make_double2(acc[mi][0], acc[mi][1]));
                }
            });
        }
        cluster_sync();
        // A22 - L21 L21^T (lower triangle) into L22
        for (int st = rank; st < kStrips; st += nranks) {
            const int i0 = st * kStrip;
            for_groups(warp, false, [&](int cg) {
                if (8 * cg >= i0 + kStrip) return;
                gemm_nt<MT>(L21 + (size_t)i0 * ld, ld, L21 + (size_t)(8 * cg) * ld, ld, 0, kN, lane, acc);
#pragma unroll
                for (int mi = 0; mi < MT; ++mi) {
                    const int i = i0 + 8 * mi + g, j = 8 * cg + 2 * t;
                    double2 v;
                    if (a.in64) {
                        v = __ldcg(reinterpret_cast<const double2*>(a.in64 + (size_t)(kN + i) * ld + kN + j));
                    } else {
                        const float2 f = *reinterpret_cast<const float2*>(a.in32 + (size_t)(kN + i) * ld + kN + j);
                        v = make_double2(f.x, f.y);
                    }
                    if (i < valid2 && j <= i) {
                        double* o = L22 + (size_t)i * ld + j;
                        if (j + 1 <= i)
                            __stcg(reinterpret_cast<double2*>(o), make_double2(v.x - acc[mi][0], v.y - acc[mi][1]));
                        else
                            __stcg(o, v.x - acc[mi][0]);
                    }
                }
            });
        }
        cluster_sync();
        // A22's chain on the first CTA; meanwhile (afterwards, when it is alone) the others
        // form T = Y11 L21^T
        if (rank == 0) chain128<true>(m, a, quadrant(a, a.L, nullptr, a.L, a.Y, kN, valid2));
        if (!a.Y) {
            for (int e = rank * kThreads + threadIdx.x; e < min(a.valid, kN) * (kN / 2); e += nranks * kThreads)
                *reinterpret_cast<double2*>(a.L + (size_t)(e / (kN / 2)) * ld + kN + 2 * (e % (kN / 2))) =
                    make_double2(0.0, 0.0);
            return;
        }
        if (nranks == 1)
            inverse_corner_t(a.Y, L21, a.T, ld, valid2, 0, 1, warp, lane);
        else if (rank != 0)
            inverse_corner_t(a.Y, L21, a.T, ld, valid2, (int)rank - 1, (int)nranks - 1, warp, lane);
        cluster_sync();
        inverse_corner_y(a.Y, a.T, ld, 0, rank, nranks, warp, lane, [&](int j, int i, double2 v) {
            // rows j of the upper right quadrant
            if (a.write_upper && j < a.valid)
                *reinterpret_cast<double2*>(a.L + (size_t)j * ld + kN + i) = make_double2(0.0, 0.0);
            if (!a.invHi) return;
            const float f[2] = {(float)v.x, (float)v.y};
#pragma unroll
            for (int q = 0; q < 2; ++q) {
                const size_t o = (size_t)(kN + i + q) * ld + j, ou = (size_t)j * ld + kN + i + q;
                a.invHi[o] = f[q];
                a.invLo[o] = tf32_low(f[q]);
                if (a.zero_upper) a.invHi[ou] = a.invLo[ou] = 0.f;
            }
        });
    }
}

// Y_k = L_kk^-T of every diagonal block k of a packed factor, one cluster a block (bsz 128:
// one CTA; bsz 256: two CTAs, one a quadrant, then Y12 over both)
template <int BSZ>
__global__ void __launch_bounds__(kThreads, 1) diag_inverse_kernel(DiagArgs a) {
    const Smem m{};
    constexpr int kQ = BSZ / kN;
    const int k = blockIdx.x / kQ;
    const int q = blockIdx.x % kQ;
    const size_t bb = (size_t)BSZ * BSZ;
    const double* L = a.in64 + (size_t)column_start(k, a.nb) * bb;
    double* Y = a.Y + (size_t)k * bb;
    const int64_t rem = a.N - (int64_t)k * BSZ - q * kN;
    const int valid = rem < 0 ? 0 : (rem < kN ? (int)rem : kN);
    chain128<false>(m, a, quadrant(a, L, nullptr, nullptr, Y, q * kN, valid));
    if constexpr (BSZ == 256) {
        const int warp = threadIdx.x >> 5, lane = threadIdx.x & 31;
        const int64_t rem2 = a.N - (int64_t)k * BSZ - kN;
        const int valid2 = rem2 < 0 ? 0 : (rem2 < kN ? (int)rem2 : kN);
        double* T = a.T + (size_t)k * kN * kN;
        cluster_sync();
        inverse_corner_t(Y, L + (size_t)kN * BSZ, T, BSZ, valid2, q, 2, warp, lane);
        cluster_sync();
        inverse_corner_y(Y, T, BSZ, 1, q, 2, warp, lane, [](int, int, double2) {});
    }
}

bool attrs_done[64] = {};
hs_status set_attrs() {
    int dev = 0;
    HS_CUDA(cudaGetDevice(&dev));
    if (dev >= 0 && dev < 64 && attrs_done[dev]) return HS_OK;
    HS_CUDA(cudaFuncSetAttribute(diag_factor_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
    HS_CUDA(cudaFuncSetAttribute(diag_factor_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
    HS_CUDA(cudaFuncSetAttribute(diag_inverse_kernel<128>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
    HS_CUDA(cudaFuncSetAttribute(diag_inverse_kernel<256>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemBytes));
    if (dev >= 0 && dev < 64) attrs_done[dev] = true;
    return HS_OK;
}

hs_status launch_cluster(void (*kernel)(DiagArgs), unsigned grid, unsigned cluster, const DiagArgs& a, cudaStream_t s) {
    cudaLaunchConfig_t cfg{};
    cfg.gridDim = dim3(grid);
    cfg.blockDim = dim3(kThreads);
    cfg.dynamicSmemBytes = kSmemBytes;
    cfg.stream = s;
    cudaLaunchAttribute at[1];
    at[0].id = cudaLaunchAttributeClusterDimension;
    at[0].val.clusterDim.x = cluster;
    at[0].val.clusterDim.y = at[0].val.clusterDim.z = 1;
    cfg.attrs = at;
    cfg.numAttrs = cluster > 1 ? 1 : 0;
    HS_CUDA(cudaLaunchKernelEx(&cfg, kernel, a));
    return HS_OK;
}

}  // namespace

hs_status launch_diag_factor(hs_ctx ctx, const DiagFactor& f, cudaStream_t s) {
    hs_status st = set_attrs();
    if (st != HS_OK) return st;
    const int bsz = ctx->bsz;
    HS_REQUIRE(bsz == 128 || bsz == 256, "the on-chip diagonal block needs matrixBlockSize 128 or 256");
    HS_REQUIRE(f.Y || (f.in_place && f.zeros), "the inverse is left out in place only");
    DiagArgs a{};
    a.in64 = f.in64;
    a.in32 = f.in32;
    a.L = f.L;
    a.pad_sqrt = f.in_place;
    a.write_upper = f.in_place && f.zeros;
    a.Y = f.Y;
    a.T = f.T;
    a.invHi = f.invHi;
    a.invLo = f.invLo;
    a.zero_upper = f.zero_upper;
    const int64_t rem = ctx->N - f.row_base;
    a.valid = rem <= 0 ? 0 : (rem < bsz ? (int)rem : bsz);
    a.info = ctx->d_info;
    a.record_neg = f.record_neg;
    a.row_base = f.row_base;
    a.ld = bsz;
    ctx->launches += 1;
    if (bsz == 128) return launch_cluster(diag_factor_kernel<128>, 1, 1, a, s);
    return launch_cluster(diag_factor_kernel<256>, (unsigned)f.ctas, (unsigned)f.ctas, a, s);
}

hs_status launch_diag_inverses(hs_ctx ctx, const double* L, double* Y, double* T, cudaStream_t s) {
    hs_status st = set_attrs();
    if (st != HS_OK) return st;
    const int bsz = ctx->bsz;
    HS_REQUIRE(bsz == 128 || bsz == 256, "the on-chip diagonal block needs matrixBlockSize 128 or 256");
    DiagArgs a{};
    a.in64 = L;
    a.Y = Y;
    a.y_full = 1;
    a.T = T;
    a.ld = bsz;
    a.nb = ctx->nb;
    a.N = ctx->N;
    ctx->launches += 1;
    if (bsz == 128) return launch_cluster(diag_inverse_kernel<128>, (unsigned)ctx->nb, 1, a, s);
    return launch_cluster(diag_inverse_kernel<256>, 2u * ctx->nb, 2, a, s);
}

hs_status launch_diag_inverse(hs_ctx ctx, const double* Lkk, double* Y, double* T, cudaStream_t s) {
    hs_status st = set_attrs();
    if (st != HS_OK) return st;
    const int bsz = ctx->bsz;
    HS_REQUIRE(bsz == 128 || bsz == 256, "the on-chip diagonal block needs matrixBlockSize 128 or 256");
    DiagArgs a{};
    a.in64 = Lkk;
    a.Y = Y;
    a.y_full = 1;
    a.T = T;
    a.ld = bsz;
    a.nb = 1;
    a.N = bsz;
    ctx->launches += 1;
    if (bsz == 128) return launch_cluster(diag_inverse_kernel<128>, 1, 1, a, s);
    return launch_cluster(diag_inverse_kernel<256>, 2, 2, a, s);
}

}  // namespace hs
