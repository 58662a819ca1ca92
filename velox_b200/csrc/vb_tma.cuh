// mbarrier and 1-D bulk-copy (TMA) helpers shared by the pipelined kernels.  Every wait is bounded.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace vb {

// The driver's tensor-map encoder, looked up once (several threads may come here first at the same time); null: it has none.
typedef CUresult (*EncodeTiledFn)(CUtensorMap*, CUtensorMapDataType, cuuint32_t, void*, const cuuint64_t*, const cuuint64_t*, const cuuint32_t*,
                                  const cuuint32_t*, CUtensorMapInterleave, CUtensorMapSwizzle, CUtensorMapL2promotion, CUtensorMapFloatOOBfill);
inline EncodeTiledFn encode_tiled_fn() {
    static const EncodeTiledFn fn = []() {
        void* p = nullptr;
        cudaDriverEntryPointQueryResult q;
        const bool ok = cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess && q == cudaDriverEntryPointSuccess;
        return ok ? reinterpret_cast<EncodeTiledFn>(p) : nullptr;
    }();
    return fn;
}

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint32_t mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok;
}
// Bounded wait (~1 s of SM clocks).  Returns false when it gave up; the caller records the failure and goes on.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 256; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (clock64() - t0 > 2000000000LL) return false;
    }
}
// The context's stop word (LaunchCfg::stop): a wait that runs out sets it, so that what was enqueued behind it does not wait its own second.
__device__ __forceinline__ bool stop_set(const uint32_t* stop) { return stop && *reinterpret_cast<const volatile uint32_t*>(stop) != 0u; }
__device__ __forceinline__ void report_wait(uint32_t* err, uint32_t* stop, uint32_t code) {
    if (err) atomicOr(err, code);
    if (stop) *reinterpret_cast<volatile uint32_t*>(stop) = code;
}
// Bounded wait of a block that goes on, and may leave, when it gives up: a second, or 10 ms where the stop word is set, which is ample for
// copies that are under way at all.
__device__ __forceinline__ bool wait_or_stop(uint32_t bar, uint32_t parity, const uint32_t* stop) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 128; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (clock64() - t0 > (stop_set(stop) ? 20000000LL : 2000000000LL)) return false;
    }
}
// Bounded wait that also gives up as soon as another thread of the block has given up (abort_flag), or the stop word is set.
constexpr uint32_t ABORT_WAITED = 1, ABORT_STOPPED = 2;
__device__ __forceinline__ bool wait_or_abort(uint32_t bar, uint32_t parity, volatile uint32_t* abort_flag, const uint32_t* stop) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long t0 = clock64();
    for (;;) {
#pragma unroll 1
        for (int i = 0; i < 128; ++i)
            if (mbar_try_wait(bar, parity)) return true;
        if (*abort_flag) return false;
        if (stop_set(stop)) { *abort_flag = ABORT_STOPPED; return false; }
        if (clock64() - t0 > 2000000000LL) { *abort_flag = ABORT_WAITED; return false; }
    }
}
// A block that gave up: what is still in flight lands before the memory that it uses is given back.  10 ms, 1 ms where only copies of its own
// first stages can be (an earlier kernel gave up: no product was started).
__device__ __forceinline__ void abort_drain(volatile uint32_t* abort_flag) {
    const long long t0 = clock64(), limit = *abort_flag == ABORT_STOPPED ? 2000000LL : 20000000LL;
    while (clock64() - t0 < limit) { }
}
// One lane of the (converged) warp, always the same one.  Tensor-core and TMA instructions take their operands from uniform
// registers: under `lane == 0` the compiler has to make them uniform instruction by instruction (the latent attention's 36
// products of a tile came 183 clocks apart instead of ~55), after elect.sync it knows that one lane runs.
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n .reg .pred p;\n elect.sync _|p, 0xFFFFFFFF;\n selp.u32 %0, 1, 0, p;\n}" : "=r"(p));
    return p != 0;
}
__device__ __forceinline__ void tma_load_1d(uint32_t dst_smem, const void* src, uint32_t bytes, uint32_t bar) {
    asm volatile("cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
                 ::"r"(dst_smem), "l"(src), "r"(bytes), "r"(bar) : "memory");
}

}  // namespace vb
