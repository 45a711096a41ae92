// Shared device helpers: shared-memory staging by bulk async copy (TMA engine,
// cp.async.bulk) completed on an mbarrier, bounded waits, status reporting.
#pragma once

#include <cstdint>
#include <string>
#include <cuda_runtime.h>

#include "../../include/disco_b200.h"

namespace disco {

// Message returned by disco_b200_last_error() for the calling thread (stored
// in a fixed per-thread buffer; the const char* form never allocates).
void set_last_error(const std::string& msg);
void set_last_error(const char* msg);

// Unique identifier of the calling thread's current context, 0 when it cannot
// be read (a device reset gives the device a new one).
unsigned long long current_context_id();

// While this lives, the thread may allocate and make or trim pools for streams
// that are not being captured although another stream is (by default such a
// call fails and ends that capture).
struct OutsideCapture {
    cudaStreamCaptureMode mode = cudaStreamCaptureModeRelaxed;
    OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    ~OutsideCapture() { cudaThreadExchangeStreamCaptureMode(&mode); }
    OutsideCapture(const OutsideCapture&) = delete;
    OutsideCapture& operator=(const OutsideCapture&) = delete;
};

// Stream-ordered scratch memory, one pool per device and context (null where
// none could be made).  32 MB (one block of the driver's) stay reserved in it, and up to 1 GB
// while a plan that has used it lives (retain gives the context whose pool it
// is, release takes it): the default pool gives
// its memory back at every synchronisation, and a call after one then pays for
// mapping it again (0.2 to 0.4 ms; 13.5 M atoms, 640 MB of scratch: 5.8 ms of an
// execute of 79).
cudaMemPool_t scratch_pool(int device);
unsigned long long scratch_retain(int device);
void scratch_release(int device, unsigned long long ctx);
int plan_create_on(const disco_loop* loops, int32_t nloops, const double box[3], const disco_options* opt,
                   int64_t max_atoms, cudaStream_t s, disco_plan** out);
// disco_b200_plan_execute, and the kernels it launched.
int plan_execute_counted(disco_plan* p, const disco_atoms* a, cudaStream_t s, int* launches);
int batch_plan_create_on(const disco_sample* samples, int32_t nsamples, const disco_options* opt, cudaStream_t s,
                         disco_batch_plan** out);
// Stream-ordered scratch of a call: from the pool, or the device's default one.
cudaError_t scratch_alloc(void** p, size_t bytes, cudaStream_t s);

// A bounded wait gives up after this many nanoseconds of %globaltimer.  A stage
// copy of a few hundred KB completes in microseconds; the bound only exists so
// that no wait can spin forever.
constexpr unsigned long long kWaitLimitNs = 2000000000ull;

__device__ __forceinline__ uint32_t smem_addr(const void* p)
{
    return static_cast<uint32_t>(__cvta_generic_to_shared(p));
}

__device__ __forceinline__ unsigned long long global_ns()
{
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count)
{
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" :: "r"(smem_addr(bar)), "r"(count) : "memory");
}

__device__ __forceinline__ void fence_mbar_init()
{
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}

__device__ __forceinline__ void fence_proxy_async_smem()
{
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}

__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t* bar, uint32_t bytes)
{
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;"
                 :: "r"(smem_addr(bar)), "r"(bytes) : "memory");
}

__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity)
{
    uint32_t ok;
    asm volatile("{\n\t.reg .pred p;\n\t"
                 "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
                 "selp.u32 %0, 1, 0, p;\n\t}"
                 : "=r"(ok) : "r"(smem_addr(bar)), "r"(parity) : "memory");
    return ok != 0;
}

// Waits for phase `parity` of the barrier; false if the bound ran out.
__device__ __forceinline__ bool mbar_wait_bounded(uint64_t* bar, uint32_t parity)
{
    if (mbar_try_wait(bar, parity)) return true;
    const unsigned long long t0 = global_ns();
    while (!mbar_try_wait(bar, parity))
        if (global_ns() - t0 > kWaitLimitNs) return false;
    return true;
}

// One bulk copy global -> shared of `bytes` (multiple of 16, both addresses
// 16-byte aligned), completing `bytes` transactions on `bar`.  Plain (no
// cluster multicast): the source is always this GPU's own memory.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 :: "r"(smem_addr(dst)), "l"(src), "r"(bytes), "r"(smem_addr(bar)) : "memory");
}

// Largest single bulk copy issued; a stage is loaded in pieces of this size.
constexpr uint32_t kBulkPiece = 65536;

// Issues the copies of one stage (called by one thread).
__device__ __forceinline__ void stage_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar)
{
    mbar_arrive_expect_tx(bar, bytes);
    for (uint32_t off = 0; off < bytes; off += kBulkPiece) {
        const uint32_t len = bytes - off < kBulkPiece ? bytes - off : kBulkPiece;
        bulk_load(static_cast<char*>(dst) + off, static_cast<const char*>(src) + off, len, bar);
    }
}

// Records the first error of a launch (first writer wins).
__device__ __forceinline__ void report(int* status, int code)
{
    atomicCAS(status, 0, code);
}

} // namespace disco
