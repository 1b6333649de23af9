// stream_common.cuh — pieces of the kernels that stream slices of packed blocks through
// shared memory (k_sweep.cu, k_cg.cu): bulk copies, bounded waits, value pairs through
// global memory, and a 32-row slice's products.
#pragma once

#include "hs_internal.cuh"
#include "tc_common.cuh"

namespace hs {
namespace {

using namespace tc;

constexpr long long kWaitClk = 4000000000ll;  // limit of a wait in SM cycles: 2 s at 2 GHz

// what the waits of a CTA share: a wait that runs out sets `fail`, and every later one returns
// at once
struct __align__(8) Waits {
    int fail;
    long long limit;  // SM cycles
};
// the same where the launch's CTAs need not be resident together from the start
struct __align__(8) ResidentWaits : Waits {
    int ctas;                  // of the launch
    const unsigned* resident;  // those counted in
};
constexpr int kAbsentLimits = 30;

// a value and its epoch, stored and read whole (16 bytes)
__device__ __forceinline__ void pair_store(ulonglong2* p, double v, unsigned long long epoch) {
    asm volatile("{\n\t.reg .b128 t;\n\tmov.b128 t, {%1, %2};\n\tst.relaxed.gpu.global.b128 [%0], t;\n\t}" ::"l"(p),
                 "l"(__double_as_longlong(v)), "l"(epoch)
                 : "memory");
}
__device__ __forceinline__ bool pair_load(const ulonglong2* p, unsigned long long epoch, double* v) {
    unsigned long long a, b;
    asm volatile("{\n\t.reg .b128 t;\n\tld.relaxed.gpu.global.b128 t, [%2];\n\tmov.b128 {%0, %1}, t;\n\t}"
                 : "=l"(a), "=l"(b)
                 : "l"(p)
                 : "memory");
    *v = __longlong_as_double(a);
    return b == epoch;
}
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];" ::"r"(
                     smem_u32(dst)),
                 "l"(src), "r"(bytes), "r"(smem_u32(bar))
                 : "memory");
}

// whether the phase is complete, without suspending the thread
__device__ __forceinline__ bool mbar_test(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.test_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}\n"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}

__device__ __forceinline__ bool out_of_time(const volatile Waits* w, long long& t0, int&) {
    return w->fail || clock64() - t0 > w->limit;
}
// The limit is meant for CTAs that run: while some of the launch are not resident, because other
// streams' kernels hold the SMs, it starts again (kAbsentLimits times at most), and once more
// when all are.  `again`: how often so far; the result: the next, or -1.
__device__ __noinline__ int begin_again(const volatile ResidentWaits* w, int again) {
    if (again == kAbsentLimits) return -1;
    return *reinterpret_cast<const volatile unsigned*>(w->resident) >= (unsigned)w->ctas ? kAbsentLimits : again + 1;
}
__device__ __forceinline__ bool out_of_time(const volatile ResidentWaits* w, long long& t0, int& again) {
    if (w->fail) return true;
    if (clock64() - t0 <= w->limit) return false;
    again = begin_again(w, again);
    t0 = clock64();
    return again < 0;
}

constexpr int kTries = 16;  // between looks at the time, which would take longer than a try
// a bounded wait by one thread.  The limit counts SM cycles: reading the global nanosecond
// timer holds up the whole SM for longer than most waits here take.
template <class W>
__device__ __forceinline__ bool thread_wait(uint64_t* bar, uint32_t parity, volatile W* w) {
    if (mbar_test(bar, parity)) return true;
    long long t0 = clock64();
    int again = 0;
    for (unsigned n = 1;; ++n) {
        if (mbar_test(bar, parity)) return true;
        if (n % kTries == 0 && out_of_time(w, t0, again)) {
            w->fail = 1;
            return false;
        }
    }
}
// the same for a whole warp, all lanes together: a wait by one lane leaves the warp split
// afterwards (its code then ran six times slower until the next row)
template <class W>
__device__ __forceinline__ bool warp_wait(uint64_t* bar, uint32_t parity, volatile W* w) {
    if (__all_sync(0xffffffffu, mbar_test(bar, parity))) return true;
    long long t0 = clock64();
    int again = 0;
    for (unsigned n = 1;; ++n) {
        if (__all_sync(0xffffffffu, mbar_test(bar, parity))) return true;
        if (n % kTries == 0 && __any_sync(0xffffffffu, out_of_time(w, t0, again))) {
            w->fail = 1;
            return false;
        }
    }
}
// Both with the thread suspended between tries: for kernels whose tensor core reads operands
// through the shared-memory port that polling warps would take.
template <class W>
__device__ __forceinline__ bool suspended_wait(uint64_t* bar, uint32_t parity, volatile W* w) {
    long long t0 = clock64();
    int again = 0;
    while (!mbar_try_wait(bar, parity)) {
        if (out_of_time(w, t0, again)) {
            w->fail = 1;
            return false;
        }
    }
    return true;
}
template <class W>
__device__ __forceinline__ bool suspended_wait_warp(uint64_t* bar, uint32_t parity, volatile W* w) {
    long long t0 = clock64();
    int again = 0;
    while (!__all_sync(0xffffffffu, mbar_try_wait(bar, parity))) {
        if (__any_sync(0xffffffffu, out_of_time(w, t0, again))) {
            w->fail = 1;
            return false;
        }
    }
    return true;
}

// Before a CTA leaves: waits until a copy in flight has landed, also after another wait has run
// out (then above all: the shared memory goes to the next CTA).  Bounded by itself.
__device__ __forceinline__ bool landed(uint64_t* bar, uint32_t parity, const volatile Waits* w) {
    const long long t0 = clock64();
    while (!mbar_test(bar, parity))
        if (clock64() - t0 > w->limit) return false;
    return true;
}

// a warp's bounded wait for a counter in global memory to reach `want`; what was written
// before it was counted up is then visible to lane 0
template <class W>
__device__ __forceinline__ bool warp_count(const unsigned long long* count, unsigned long long want, int lane,
                                           volatile W* w) {
    long long t0 = clock64();
    int again = 0;
    for (;;) {
        unsigned long long have = 0;
        if (lane == 0) asm volatile("ld.acquire.gpu.global.u64 %0, [%1];" : "=l"(have) : "l"(count) : "memory");
        if (__shfl_sync(0xffffffffu, have, 0) >= want) return true;
        if (__any_sync(0xffffffffu, out_of_time(w, t0, again))) {
            w->fail = 1;
            return false;
        }
    }
}

// lane l's pairs p[l + 32 q], q < M, once they carry the epoch; bounded as above.  While
// they do not, only the last of each 32 is polled, and not at full rate: over a hundred CTAs
// wait for the same vector, and polling all of it slowed the chain sixfold.
template <int M, class W>
__device__ __forceinline__ bool warp_pairs(const ulonglong2* p, unsigned long long epoch, int lane, volatile W* w,
                                           int* err, double (&v)[M]) {
    long long t0 = clock64();
    int again = 0;
    for (int n = 0;; ++n) {
        double one;
        bool done = lane >= M || pair_load(p + 32 * (lane % M) + 31, epoch, &one);
        if (__all_sync(0xffffffffu, done)) {
#pragma unroll
            for (int q = 0; q < M; ++q) done &= pair_load(p + lane + 32 * q, epoch, &v[q]);
            if (__all_sync(0xffffffffu, done)) return true;
        }
        if ((n & 63) == 63 &&
            __any_sync(0xffffffffu, out_of_time(w, t0, again) || *reinterpret_cast<volatile int*>(err) != 0)) {
            w->fail = 1;
            return false;
        }
        __nanosleep(40);
    }
}

// A slice of a block in shared memory: COLS false: 32 rows of BSZ, row major (output o =
// row 4 warp + o); COLS true: BSZ rows of 32 columns in boxes of 128-byte rows with the
// 128-byte swizzle (output o = column 4 warp + o, the block's transposed product).  A
// thread holds BSZ / 8 of its values; its part of the warp's 4 outputs in s[], and of the
// vector the entries at index().
template <int BSZ, typename T, bool COLS>
struct Slice {
    static constexpr int kV = 16 / (int)sizeof(T);  // values a 16-byte load
    static constexpr int kLoads = BSZ / 8 / kV;

    static __device__ __forceinline__ void load(const uint8_t* tile, int warp, int lane, T (&v)[BSZ / 8]) {
#pragma unroll
        for (int q = 0; q < kLoads; ++q) {
            const uint8_t* p;
            if constexpr (!COLS) {  // rows first: q = row * loads a row + m
                constexpr int kM = kLoads / 4;
                p = tile + ((size_t)(4 * warp + q / kM) * BSZ + ((q % kM) * 32 + lane) * kV) * sizeof(T);
            } else if constexpr (sizeof(T) == 8) {  // 2 boxes of 16 columns; lane: column pair lane / 16, row lane % 16 + 16 q
                const int r = (lane & 15) + 16 * q, ch = (warp & 3) * 2 + (lane >> 4);
                p = tile + (size_t)(warp >> 2) * BSZ * 128 + r * 128 + ((ch ^ (r & 7)) << 4);
            } else {  // one box of 32 columns; lane: row lane + 32 q
                const int r = lane + 32 * q;
                p = tile + r * 128 + ((warp ^ (r & 7)) << 4);
            }
            if constexpr (sizeof(T) == 8) {
                const double2 d = *reinterpret_cast<const double2*>(p);
                v[2 * q] = d.x;
                v[2 * q + 1] = d.y;
            } else {
                const float4 f = *reinterpret_cast<const float4*>(p);
                v[4 * q] = f.x;
                v[4 * q + 1] = f.y;
                v[4 * q + 2] = f.z;
                v[4 * q + 3] = f.w;
            }
        }
    }

    // s[o] += part of the products with the vector x (shared memory)
    static __device__ __forceinline__ void apply(const T (&v)[BSZ / 8], const double* x, int lane, double (&s)[4]) {
        if constexpr (!COLS) {
            constexpr int kM = kLoads / 4;
#pragma unroll
            for (int m = 0; m < kM; ++m) {
                double xv[kV];
#pragma unroll
                for (int e = 0; e < kV; e += 2) {
                    const double2 d = *reinterpret_cast<const double2*>(x + (m * 32 + lane) * kV + e);
                    xv[e] = d.x;
                    xv[e + 1] = d.y;
                }
#pragma unroll
                for (int o = 0; o < 4; ++o)
#pragma unroll
                    for (int e = 0; e < kV; ++e) s[o] = fma((double)v[(o * kM + m) * kV + e], xv[e], s[o]);
            }
        } else if constexpr (sizeof(T) == 8) {  // s[0], s[1]: columns 2 (lane / 16) + {0, 1}
#pragma unroll
            for (int q = 0; q < kLoads; ++q) {
                const double xr = x[(lane & 15) + 16 * q];
                s[0] = fma((double)v[2 * q], xr, s[0]);
                s[1] = fma((double)v[2 * q + 1], xr, s[1]);
            }
        } else {
#pragma unroll
            for (int q = 0; q < kLoads; ++q) {
                const double xr = x[lane + 32 * q];
#pragma unroll
                for (int o = 0; o < 4; ++o) s[o] = fma((double)v[4 * q + o], xr, s[o]);
            }
        }
    }

    // the total of output lane / 8
    static __device__ __forceinline__ double total(const double (&s)[4], int lane) {
        const bool b3 = lane & 8, b4 = lane & 16;
        double a;
        if constexpr (COLS && sizeof(T) == 8) {
            a = (b3 ? s[1] : s[0]) + __shfl_xor_sync(0xffffffffu, b3 ? s[0] : s[1], 8);
        } else {
            const double a0 = (b4 ? s[2] : s[0]) + __shfl_xor_sync(0xffffffffu, b4 ? s[0] : s[2], 16);
            const double a1 = (b4 ? s[3] : s[1]) + __shfl_xor_sync(0xffffffffu, b4 ? s[1] : s[3], 16);
            a = (b3 ? a1 : a0) + __shfl_xor_sync(0xffffffffu, b3 ? a0 : a1, 8);
        }
        a += __shfl_xor_sync(0xffffffffu, a, 4);
        a += __shfl_xor_sync(0xffffffffu, a, 2);
        a += __shfl_xor_sync(0xffffffffu, a, 1);
        return a;
    }
};

}  // namespace
}  // namespace hs
