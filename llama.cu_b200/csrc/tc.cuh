// tcgen05 / TMEM / TMA / mbarrier helpers shared by the 5th-generation tensor-core kernels, and the tensor-map encoder.
#pragma once
#include <cuda.h>

#include <mutex>

#include "common.cuh"

namespace lcu {

#ifdef __CUDACC__
constexpr unsigned long long TC_WAIT_NS = 2000000000ull;
__device__ __forceinline__ unsigned long long tc_ns() {
    unsigned long long t;
    asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t));
    return t;
}
__device__ __forceinline__ uint32_t tc_smem(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ void tc_mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void tc_mbar_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(bar), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool tc_mbar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile("{\n .reg .pred p;\n mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n selp.u32 %0, 1, 0, p;\n}"
                 : "=r"(ok) : "r"(bar), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ bool tc_mbar_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    if (tc_mbar_try(bar, parity)) return true;
    unsigned long long t0 = tc_ns();
    for (unsigned it = 1;; ++it) {
        if (tc_mbar_try(bar, parity)) return true;
        if ((it & 255u) == 0 && (*abort_flag || tc_ns() - t0 > TC_WAIT_NS)) return false;
    }
}
// ---- After a wait has run out a CTA may leave only when nothing writes to its memory any more: its copies have landed and its MMAs
// have ended.  A barrier that stays open (an arrival that never came) ends by a limit far above what a copy takes.
constexpr unsigned long long TC_DRAIN_NS = 10000000ull;
__device__ __forceinline__ void tc_warp_drain(uint32_t bar, uint32_t parity) {
    const unsigned long long t0 = tc_ns();
    while (!__all_sync(0xffffffffu, tc_mbar_try(bar, parity)) && __all_sync(0xffffffffu, tc_ns() - t0 < TC_DRAIN_NS)) {
    }
}
// a ring of `stages` barriers that was filled `issued` times: only the last fill of a stage can be open
__device__ __forceinline__ void tc_warp_drain_ring(uint32_t full0, int issued, int stages) {
    for (int f = issued > stages ? issued - stages : 0; f < issued; ++f) tc_warp_drain(full0 + 8 * (f % stages), (uint32_t)(f / stages) & 1u);
}
// ---- forms for a whole converged warp: one elected lane issues, and nothing but the instruction depends on the lane, so the
// compiler keeps operands and loop in uniform registers (issued from a `lane == 0` branch, four MMAs take 270 cycles to issue)
__device__ __forceinline__ bool tc_warp_wait(uint32_t bar, uint32_t parity, volatile int *abort_flag) {
    if (__all_sync(0xffffffffu, tc_mbar_try(bar, parity))) return true;
    return __all_sync(0xffffffffu, tc_mbar_wait(bar, parity, abort_flag));
}
__device__ __forceinline__ void tc_warp_expect_tx(uint32_t bar, uint32_t bytes) {
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n @e mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;\n}" ::"r"(bar), "r"(bytes) : "memory");
}
// a K block of 64: four MMAs of K = 16 on operand tiles with 128-byte swizzle
#define LCU_TC_MMA4(GROUP)                                                                                                          \
    "{\n .reg .pred e, p, q;\n .reg .b64 a, b;\n elect.sync _|e, 0xffffffff;\n setp.ne.b32 p, %4, 0;\n setp.eq.b32 q, 0, 0;\n"       \
    " @e tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], %1, %2, %3, p;\n add.u64 a, %1, 2;\n add.u64 b, %2, 2;\n"               \
    " @e tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], a, b, %3, q;\n add.u64 a, %1, 4;\n add.u64 b, %2, 4;\n"                 \
    " @e tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], a, b, %3, q;\n add.u64 a, %1, 6;\n add.u64 b, %2, 6;\n"                 \
    " @e tcgen05.mma.cta_group::" GROUP ".kind::f16 [%0], a, b, %3, q;\n}"
__device__ __forceinline__ void tc_warp_mma4(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile(LCU_TC_MMA4("1") ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_warp_commit(uint32_t bar) {
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n @e tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];\n}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_warp_tma_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("{\n .reg .pred e;\n elect.sync _|e, 0xffffffff;\n"
                 " @e cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];\n}"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
__device__ __forceinline__ void tc_tma_2d(uint32_t dst, const CUtensorMap *map, int x, int y, uint32_t bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(x), "r"(y), "r"(bar) : "memory");
}
// shared-memory operand descriptor: K-major tile, 128-byte swizzle, 8-row groups 1024 bytes apart
__device__ __forceinline__ uint64_t tc_desc(uint32_t saddr) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | (1ull << 16) | (64ull << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tc_mma_f16(uint32_t d_tmem, uint64_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n .reg .pred p;\n setp.ne.b32 p, %4, 0;\n tcgen05.mma.cta_group::1.kind::f16 [%0], %1, %2, %3, p;\n}"
                 ::"r"(d_tmem), "l"(a), "l"(b), "r"(idesc), "r"(accumulate) : "memory");
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ void tc_ld16(uint32_t taddr, uint32_t r[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]), "=r"(r[8]),
                   "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}

__device__ __forceinline__ void tc_ld8(uint32_t taddr, uint32_t r[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr) : "memory");
}
#endif  // __CUDACC__

typedef CUresult (*TcEncodeFn)(CUtensorMap *, CUtensorMapDataType, cuuint32_t, void *, const cuuint64_t *, const cuuint64_t *,
                               const cuuint32_t *, const cuuint32_t *, CUtensorMapInterleave, CUtensorMapSwizzle,
                               CUtensorMapL2promotion, CUtensorMapFloatOOBfill);

inline TcEncodeFn tc_encode_fn() {
    static TcEncodeFn fn = nullptr;
    static bool tried = false;
    static std::mutex mu;
    std::lock_guard<std::mutex> lk(mu);
    if (!tried) {
        tried = true;
        void *p = nullptr;
        cudaDriverEntryPointQueryResult q;
        if (cudaGetDriverEntryPoint("cuTensorMapEncodeTiled", &p, cudaEnableDefault, &q) == cudaSuccess &&
            q == cudaDriverEntryPointSuccess)
            fn = reinterpret_cast<TcEncodeFn>(p);
    }
    return fn;
}

}  // namespace lcu
