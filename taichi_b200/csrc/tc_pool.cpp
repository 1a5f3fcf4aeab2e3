// tc_pool.cpp -- scratch memory of plan and format builds, stream-ordered.
//
// A build needs a dozen device arrays for a few milliseconds.  cudaMalloc and
// cudaFree cost 340 + 270 us a pair on a B200 host whatever the size (the
// free waits for the device), which was most of a build; an allocation from a
// pool that still holds the memory of the last build costs 2 us.  So scratch
// comes from a memory pool of the library's own (not the device's default
// pool, whose settings belong to the program), one per device.  It keeps at
// most kPoolKeep bytes between builds: it lets go of more at the wait that
// ends a call, after the call's scratch is freed (ScratchEnd).  It gives all
// but kPoolIdle of them back when the process's last plan is destroyed (in
// the device that is current then); a plan that finds no room takes all of
// them back first.  The pool is found by the CUDA context it was made
// in, so a device reset starts a new one.  Allocations and frees are ordered
// on the build's own stream; pools are safe across threads and streams.

#include <cuda.h>
#include <cuda_runtime.h>

#include <algorithm>
#include <atomic>
#include <mutex>

#include "tc_ctxcache.h"
#include "tc_internal.h"

namespace tc {
namespace {

constexpr size_t kPoolKeep = 256u << 20;
// What stays after the last plan: a program that makes and drops one plan at
// a time does not pay for unmapping (0.3 ms, and hundreds at times when other
// processes use the machine's driver) and mapping with every plan.
constexpr size_t kPoolIdle = 64u << 20;

ContextAddressCache<> g_pools;
std::atomic<long> g_live_plans{0};

// The library's pool in the current context, or null when there is none and
// plain allocations are to be used.  make: create it if it is missing.
cudaMemPool_t current_pool(bool make)
{
    int dev = 0;
    if (cudaGetDevice(&dev) != cudaSuccess) return nullptr;
    unsigned long long ctx = current_context_id();
    if (ctx == 0 && make && cudaSetDevice(dev) == cudaSuccess) ctx = current_context_id();   // first use here
    if (ctx == 0) return nullptr;               // cannot be told from another context's
    void *p = nullptr;
    const int rc = g_pools.get(dev, ctx, [&](void **out) {
        if (!make) return 1;
        cudaMemPoolProps props{};
        props.allocType = cudaMemAllocationTypePinned;
        props.location.type = cudaMemLocationTypeDevice;
        props.location.id = dev;
        cudaMemPool_t pool = nullptr;
        if (cudaMemPoolCreate(&pool, &props) != cudaSuccess) return 1;
        uint64_t keep = kPoolKeep;
        if (cudaMemPoolSetAttribute(pool, cudaMemPoolAttrReleaseThreshold, &keep) != cudaSuccess) {
            cudaMemPoolDestroy(pool);
            return 1;
        }
        *out = pool;
        return 0;
    }, &p);
    if (rc != 0) {
        (void)cudaGetLastError();
        return nullptr;
    }
    return static_cast<cudaMemPool_t>(p);
}

}  // namespace

unsigned long long current_context_id()
{
    using GetCurrent = CUresult (*)(CUcontext *);
    using GetId = CUresult (*)(CUcontext, unsigned long long *);
    static GetCurrent get_current = nullptr;
    static GetId get_id = nullptr;
    static std::once_flag once;
    std::call_once(once, [] {
        void *a = nullptr, *b = nullptr;
        cudaDriverEntryPointQueryResult qa, qb;
        if (cudaGetDriverEntryPoint("cuCtxGetCurrent", &a, cudaEnableDefault, &qa) == cudaSuccess &&
            cudaGetDriverEntryPoint("cuCtxGetId", &b, cudaEnableDefault, &qb) == cudaSuccess &&
            qa == cudaDriverEntryPointSuccess && qb == cudaDriverEntryPointSuccess) {
            get_current = reinterpret_cast<GetCurrent>(a);
            get_id = reinterpret_cast<GetId>(b);
        }
        (void)cudaGetLastError();
    });
    if (!get_current || !get_id) return 0;
    CUcontext ctx = nullptr;
    unsigned long long id = 0;
    if (get_current(&ctx) != CUDA_SUCCESS || !ctx || get_id(ctx, &id) != CUDA_SUCCESS) return 0;
    return id;
}

Scratch::~Scratch() { release(); }

ScratchEnd::~ScratchEnd()
{
    if (on) cudaStreamSynchronize(s);
}

void Scratch::release()
{
    if (!p) return;
    if (pooled) cudaFreeAsync(p, s);
    else cudaFree(p);
    p = nullptr;
}

tc_status Scratch::alloc(size_t bytes, cudaStream_t stream)
{
    release();
    bytes = std::max<size_t>(bytes, 16);
    s = stream;
    cudaMemPool_t pool = current_pool(true);
    pooled = pool && cudaMallocFromPoolAsync(&p, bytes, pool, stream) == cudaSuccess;
    if (pooled) return TC_OK;
    (void)cudaGetLastError();
    return device_alloc(&p, bytes, stream);
}

tc_status device_alloc(void **p, size_t bytes, cudaStream_t stream)
{
    cudaError_t e = cudaMalloc(p, bytes);
    if (e != cudaSuccess) {               // once more without what the pool holds unused
        (void)cudaGetLastError();
        if (cudaMemPool_t pool = current_pool(false)) {
            if (cudaStreamSynchronize(stream) == cudaSuccess) cudaMemPoolTrimTo(pool, 0);
            e = cudaMalloc(p, bytes);
        }
    }
    if (e == cudaSuccess) return TC_OK;
    (void)cudaGetLastError();
    *p = nullptr;
    return fail(TC_ERR_ALLOC, "cudaMalloc(%zu): %s", bytes, cudaGetErrorString(e));
}

tc_status upload(void *dst, const void *src, size_t bytes)
{
    TC_CUDA(cudaMemcpy(dst, src, bytes, cudaMemcpyHostToDevice));
    TC_CUDA(cudaStreamSynchronize(nullptr));
    return TC_OK;
}

void plan_born() { g_live_plans.fetch_add(1, std::memory_order_relaxed); }

void plan_gone()
{
    if (g_live_plans.fetch_sub(1, std::memory_order_relaxed) != 1) return;
    if (cudaMemPool_t pool = current_pool(false)) cudaMemPoolTrimTo(pool, kPoolIdle);
    (void)cudaGetLastError();
}

}  // namespace tc
