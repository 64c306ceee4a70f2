// Host logic of the tensor kernels' plans when a CUDA call fails, without a GPU: the runtime's calls are
// wrapped (-Wl,--wrap) by a fake that keeps "device" memory on the host, launches nothing and fails the
// k-th call on demand.  For every k: what another search may be reading stays, nothing that was begun
// is taken for made, a second try completes, and at the end nothing is left allocated.
#include <atomic>
#include <cstdio>
#include <cstdlib>
#include <cstring>
#include <mutex>
#include <set>
#include <thread>
#include <vector>

#include "ctx.h"
#include "tensor3x.h"

static std::set<void*> live;
static std::mutex fake_mu;  // (the last scenario has several threads)
static std::atomic<long> calls{0}, fail_at{0}, launches{0}, maps{0};
static bool failing() { return ++calls == fail_at; }
#define CHECK(c) do { if (!(c)) { std::printf("%s:%d: %s (fail_at %ld)\n", __FILE__, __LINE__, #c, fail_at.load()); std::exit(1); } } while (0)

static CUresult encode(CUtensorMap* m, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*,
                       const cuuint32_t*, const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle,
                       CUtensorMapL2promotion, CUtensorMapFloatOOBfill) {
    if (failing()) return CUDA_ERROR_INVALID_VALUE;
    std::memset(m, 0x5a, sizeof(*m));
    ++maps;
    return CUDA_SUCCESS;
}
extern "C" {
cudaError_t __wrap_cudaMalloc(void** p, size_t n) {
    if (failing()) return cudaErrorMemoryAllocation;
    std::this_thread::yield();
    std::lock_guard<std::mutex> g(fake_mu);
    *p = std::calloc(1, n ? n : 1);
    live.insert(*p);
    return cudaSuccess;
}
cudaError_t __wrap_cudaFree(void* p) {
    if (!p) return cudaSuccess;
    std::lock_guard<std::mutex> g(fake_mu);
    CHECK(live.erase(p) == 1);
    std::free(p);
    return cudaSuccess;
}
cudaError_t __wrap_cudaMemcpy(void* d, const void* s, size_t n, cudaMemcpyKind) {
    if (failing()) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t __wrap_cudaMemcpyAsync(void* d, const void* s, size_t n, cudaMemcpyKind, cudaStream_t) {
    if (failing()) return cudaErrorUnknown;
    std::memcpy(d, s, n);
    return cudaSuccess;
}
cudaError_t __wrap_cudaStreamSynchronize(cudaStream_t) { return failing() ? cudaErrorUnknown : cudaSuccess; }
cudaError_t __wrap_cudaGetLastError() { return failing() ? cudaErrorUnknown : cudaSuccess; }
cudaError_t __wrap_cudaLaunchKernel(const void*, dim3, dim3, void**, size_t, cudaStream_t) {
    ++launches;
    return cudaSuccess;
}
cudaError_t __wrap___cudaLaunchKernel(cudaKernel_t, dim3, dim3, void**, size_t, cudaStream_t) {
    ++launches;
    return cudaSuccess;
}
cudaError_t __wrap_cudaFuncSetAttribute(const void*, cudaFuncAttribute, int) { return cudaSuccess; }
cudaError_t __wrap_cudaOccupancyMaxActiveClusters(int* n, const void*, const cudaLaunchConfig_t*) {
    *n = 76;
    return cudaSuccess;
}
cudaError_t __wrap_cudaOccupancyMaxActiveBlocksPerMultiprocessorWithFlags(int* n, const void*, int, size_t, unsigned) {
    *n = 1;
    return cudaSuccess;
}
cudaError_t __wrap_cudaGetDriverEntryPointByVersion(const char*, void** p, unsigned, unsigned long long,
                                                    cudaDriverEntryPointQueryResult* q) {
    *p = (void*)encode;
    *q = cudaDriverEntryPointSuccess;
    return cudaSuccess;
}
}

using namespace fiu;

static const DevData kData{nullptr, nullptr, nullptr, 40, 5, 5, 300, 290};
static const uint4* kPairs = reinterpret_cast<const uint4*>(0x1000);  // not read: nothing is launched

// Runs `make` with every one of its CUDA calls failing in turn and `kept` checked after each, then again without.
template <class Make, class Kept>
static void each_failure(Make&& make, Kept&& kept) {
    for (long k = 1;; ++k) {
        calls = 0;
        fail_at = k;
        const int e = make();
        const bool reached = calls >= k;
        fail_at = 0;
        if (!reached) {
            CHECK(e == 0);
            return;
        }
        CHECK(e != 0);
        kept();
    }
}

static void whole_scans() {
    T3Plan plan;
    tensor3_prepare(kData, plan);
    each_failure([&] { return (int)tensor3_order_items(plan, kData, 2, nullptr, nullptr, 152); },
                 [&] { CHECK(!plan.f4.ones || maps >= 2); });
    uint8_t* ones = plan.f4.ones;
    CHECK(ones && live.count(ones) && plan.item2_begin);
    each_failure([&] { return (int)tensor3_order_items(plan, kData, 3, nullptr, nullptr, 152); },
                 [&] { CHECK(plan.f4.ones == ones && live.count(ones)); });
    CHECK(plan.f4.bits && plan.f4.ones == ones && live.count(ones));
    each_failure([&] { return (int)tensor3_order_items(plan, kData, 4, kPairs, nullptr, 152); },
                 [&] { CHECK(plan.f4.ones == ones && live.count(ones) && plan.f4.bits); });
    CHECK(plan.f4.tri && plan.item4_begin && plan.item4_per);
    tensor3_release(plan);
    CHECK(live.empty());
}

static void layers() {
    T3Plan plan;
    tensor3_prepare(kData, plan);
    ScanWork w{};
    w.d = kData;
    w.dist_n = kData.snps;
    w.dist_step = 3;
    w.dist_offset = 1;
    for (w.order = 2; w.order <= 4; ++w.order)
        each_failure([&] { return (int)tensor3_layer(plan, w, kPairs, nullptr, 152); },
                     [&] { CHECK(tensor_units(plan, w) == 0); });
    tensor3_release(plan);
    CHECK(live.empty());
}

static void core_tables() {
    fiu_ctx ctx;
    ctx.sms = 152;
    fiu_resident r;
    r.d = kData;
    r.one_hot = 1;
    int kernel = 0;
    each_failure([&] { return choose_kernel(&ctx, &r, 2, FIU_KERNEL_ELIDED_HS, kernel); }, [&] { CHECK(!r.single); });
    uint32_t* single = r.single;
    CHECK(live.count(single) && !r.pairs);
    each_failure([&] { return choose_kernel(&ctx, &r, 4, FIU_KERNEL_ELIDED_POPC, kernel); },
                 [&] { CHECK(r.single == single && live.count(single) && !r.pairs && !r.triples); });
    CHECK(r.single == single && live.count(r.pairs) && live.count(r.triples) && live.size() == 3);
    for (void* p : {(void*)r.single, (void*)r.pairs, (void*)r.triples}) __wrap_cudaFree(p);
    CHECK(live.empty());
}

// Several contexts make the tables, plan and layer of one data set at once: each is made once.
static void at_once() {
    for (int round = 0; round < 200; ++round) {
        fiu_resident r;
        r.d = kData;
        r.one_hot = 1;
        std::vector<std::thread> threads;
        std::vector<int> rc(4, -1);
        for (int t = 0; t < 4; ++t)
            threads.emplace_back([&, t] {
                fiu_ctx ctx;
                ctx.sms = 152;
                ScanWork w{};
                w.d = kData;
                w.order = 2 + t % 3;
                w.dist_n = kData.snps;
                w.dist_step = t == 3 ? 3 : 1;
                int kernel = 0, tp = 0;
                rc[t] = choose_tile(&ctx, &r, w, FIU_KERNEL_AUTO, kernel, tp, Use::kSearch);
            });
        for (std::thread& t : threads) t.join();
        for (int e : rc) CHECK(e == FIU_OK);
        CHECK(r.single && r.pairs && r.t3);
        tensor3_release(*r.t3);
        delete r.t3;
        __wrap_cudaFree(r.single);
        __wrap_cudaFree(r.pairs);
        CHECK(live.empty());
    }
}

int main() {
    whole_scans();
    layers();
    core_tables();
    at_once();
    std::printf("ok\n");
}
