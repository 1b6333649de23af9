// k_selftest.cu — self-test of the bounded device-side waits: every wait that the library's
// kernels use, on something that never happens, with a short limit; and the wait for copies in
// flight before a CTA leaves, after another wait has run out.  No reference counterpart.
#include <climits>
#include <string>

#include "hs_internal.cuh"
#include "stream_common.cuh"

namespace hs {
namespace {

// one warp a wait
enum { kThread, kWarp, kSuspended, kSuspendedWarp, kCount, kPairs, kTimer, kLanded, kAbsent, kResident, kWaitKinds };
const char* const kNames[kWaitKinds] = {"thread_wait", "warp_wait",  "suspended_wait", "suspended_wait_warp",
                                        "warp_count",  "warp_pairs", "mbar_wait_for",  "landed",
                                        "warp_wait with absent CTAs", "warp_wait with all CTAs"};
constexpr int kCopyBytes = 16384;

struct SelftestArgs {
    long long limit;                  // SM cycles
    unsigned long long limit_ns;
    const unsigned long long* count;  // zero
    const ulonglong2* pairs;          // 32, zero
    const unsigned* source;           // kCopyBytes of 0x5a
    int* err;
    int* ran_out;                     // [wait]: 1 if it ran out, and the next one returned at once
    long long* info;                  // the trailing update's mark
};

__global__ void __launch_bounds__(32) wait_selftest_kernel(SelftestArgs a) {
    __shared__ __align__(16) unsigned copied[kCopyBytes / 4];
    __shared__ uint64_t bar, loaded;
    __shared__ ResidentWaits s_waits;
    volatile Waits* waits = &s_waits;
    const int lane = threadIdx.x, kind = blockIdx.x;
    if (lane == 0) {
        mbar_init(&bar, 1);  // nothing arrives
        mbar_init(&loaded, 1);
        fence_barrier_init();
        s_waits.fail = 0;
        s_waits.limit = kind < kAbsent ? a.limit : a.limit / (kAbsentLimits + 1);
        s_waits.resident = reinterpret_cast<const unsigned*>(a.count);  // zero
        s_waits.ctas = kind == kAbsent ? 1 : 0;
    }
    __syncwarp();
    auto wait = [&]() -> bool {
        double v[1];
        switch (kind) {
            case kThread: return lane != 0 || thread_wait(&bar, 0, waits);
            case kWarp: return warp_wait(&bar, 0, waits);
            case kSuspended: return lane != 0 || suspended_wait(&bar, 0, waits);
            case kSuspendedWarp: return suspended_wait_warp(&bar, 0, waits);
            case kCount: return warp_count(a.count, 1, lane, waits);
            case kPairs: return warp_pairs(a.pairs, 1, lane, waits, a.err, v);
            default: return lane != 0 || mbar_wait_for(&bar, 0, a.limit_ns);
        }
    };
    if (kind == kLanded) {
        // a copy still in flight when a wait has run out is waited for all the same, and what
        // never lands is not waited for without end
        if (lane == 0) {
            s_waits.fail = 1;
            mbar_arrive_expect_tx(&loaded, kCopyBytes);
            bulk_load(copied, a.source, kCopyBytes, &loaded);
        }
        __syncwarp();
        bool in = landed(&loaded, 0, waits);
        for (int e = lane; e < kCopyBytes / 4; e += 32) in = in && copied[e] == 0x5a5a5a5au;
        const long long t0 = clock64();
        in = __all_sync(0xffffffffu, in && !landed(&bar, 0, waits) && clock64() - t0 > a.limit);
        if (lane == 0) a.ran_out[kind] = in;
        return;
    }
    if (kind >= kAbsent) {
        // the limit again and again for CTAs that are absent, once more when all are there
        const long long t0 = clock64();
        bool out = !warp_wait(&bar, 0, static_cast<volatile ResidentWaits*>(&s_waits));
        const long long limits = (clock64() - t0) / s_waits.limit;
        out = out && (kind == kAbsent ? limits > kAbsentLimits : limits >= 2 && limits < kAbsentLimits / 2);
        if (lane == 0) a.ran_out[kind] = out;
        return;
    }
    bool out = !wait();
    __syncwarp();
    if (kind != kTimer) {
        const long long t0 = clock64();
        out = out && !wait() && clock64() - t0 < a.limit / 2 && waits->fail == 1;
        if (lane == 0 && out && (kind == kSuspended || kind == kSuspendedWarp)) atomicMin(a.info, -1ll);
    }
    if (lane == 0) a.ran_out[kind] = out;
}

}  // namespace

hs_status launch_bounded_wait_selftest(hs_ctx ctx, int64_t timeout_ns) {
    hs_status st = ensure_scratch(ctx, kSmallScratch);
    if (st != HS_OK) return st;
    cudaStream_t s = ctx->stream;
    char* base = static_cast<char*>(ctx->scratch);
    SelftestArgs a{};
    a.limit = 2 * timeout_ns;  // the SM clock stays below 2 GHz
    a.limit_ns = (unsigned long long)timeout_ns;
    a.ran_out = reinterpret_cast<int*>(base);
    a.count = reinterpret_cast<unsigned long long*>(base + 256);
    a.err = reinterpret_cast<int*>(base + 512);
    a.pairs = reinterpret_cast<ulonglong2*>(base + 1024);
    a.source = reinterpret_cast<unsigned*>(base + 4096);
    a.info = ctx->d_info;
    // the pivot record is lent to the test
    long long record = 0;
    HS_CUDA(cudaMemcpyAsync(&record, ctx->d_info, sizeof(record), cudaMemcpyDeviceToHost, s));
    HS_CUDA(cudaMemsetAsync(base, 0, 4096, s));
    HS_CUDA(cudaMemsetAsync(base + 4096, 0x5a, kCopyBytes, s));
    HS_CUDA(cudaStreamSynchronize(s));
    set_i64_dev(ctx->d_info, INT64_MAX, s);
    ctx->launches += 2;
    wait_selftest_kernel<<<kWaitKinds, 32, 0, s>>>(a);
    HS_CHECK_LAUNCH("wait_selftest");
    int out[kWaitKinds];
    HS_CUDA(cudaMemcpyAsync(out, a.ran_out, sizeof(out), cudaMemcpyDeviceToHost, s));
    HS_CUDA(cudaStreamSynchronize(s));
    const hs_status mark = hs_ctx_take_info(ctx, nullptr);
    set_i64_dev(ctx->d_info, record, s);
    HS_CHECK_LAUNCH("restore info");
    std::string names, wrong;
    for (int i = 0; i < kWaitKinds; ++i) {
        std::string& list = out[i] ? names : wrong;
        list += (list.empty() ? "" : ", ") + std::string(kNames[i]);
    }
    if (!wrong.empty()) {
        set_error("hs_selftest_bounded_wait: these waits did not run out: " + wrong);
        return HS_OK;
    }
    if (mark != HS_ERR_TIMEOUT) {
        set_error("hs_selftest_bounded_wait: the trailing update's mark was not reported");
        return HS_ERR_CUDA;
    }
    set_error("hs_selftest_bounded_wait: every bounded wait ran out, as expected here: " + names);
    return HS_ERR_TIMEOUT;
}

}  // namespace hs
