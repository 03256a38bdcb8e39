// Inline-PTX wrappers for the sm_100a asynchronous machinery the kernels share: mbarriers with bounded
// waits, TMA (tiled and plain bulk) copies, and the tcgen05 tensor-memory instructions.
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

#include "mlxq_device.cuh"

namespace mlxq {

constexpr uint64_t WAIT_NS = 2000000000ull;   // 2 s per wait before giving up

// ---- PTX wrappers ---------------------------------------------------------------------------------------
__device__ __forceinline__ uint32_t smem_u32(const void* p) { return static_cast<uint32_t>(__cvta_generic_to_shared(p)); }

__device__ __forceinline__ void mbar_init(uint64_t* bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t* bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
__device__ __forceinline__ void mbar_expect_tx(uint64_t* bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t* bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok) : "r"(smem_u32(bar)), "r"(parity) : "memory");
    return ok != 0;
}
__device__ __forceinline__ uint64_t global_ns() {
    uint64_t t;
    asm volatile("mov.u64 %0, %globaltimer;" : "=l"(t));
    return t;
}

// Bounded wait.  Returns false when the CTA is aborting (this wait ran out, or another role's did).
static __device__ __noinline__ bool mbar_wait_slow(uint64_t* bar, uint32_t parity, int* abort_flag, unsigned* err) {
    const uint64_t t0 = global_ns();
    for (;;) {
        for (int i = 0; i < 64; i++)
            if (mbar_try_wait(bar, parity)) return true;       // (a __nanosleep between tries: no gain for the GEMM, 5 % loss for decode)
        if (*reinterpret_cast<volatile int*>(abort_flag)) return false;
        if (global_ns() - t0 > WAIT_NS) {
            *reinterpret_cast<volatile int*>(abort_flag) = 1;
            atomicOr(err, ERR_WAIT_TIMEOUT | ERR_GEMM_PIPELINE);
            return false;
        }
    }
}
__device__ __forceinline__ bool mbar_wait(uint64_t* bar, uint32_t parity, int* abort_flag, unsigned* err) {
    if (mbar_try_wait(bar, parity)) return true;
    return mbar_wait_slow(bar, parity, abort_flag, err);
}

// Whole-warp wait for code that goes on to a ".sync.aligned" instruction (tcgen05.ld / tcgen05.st / mma.sync).
// Lane 0 polls alone (bounded, like mbar_wait) and the result is broadcast; __syncwarp orders the other lanes'
// later reads after lane 0's acquire.  Must be called by all 32 lanes.
//
// Why one lane.  With every lane running its own mbar_wait before a tcgen05.st, the store now and then lost the
// data of some lanes (measured on B200, at full GEMM size only).  Read against the PTX rules, the all-lanes form
// was in order on three counts: the phase parity is computed from warp-uniform counters, so no lane can wait for a
// different phase; the barrier cannot advance twice while a lane of the warp still waits (the next phase needs this
// warp's own arrival on full_a); and tcgen05.fence::after_thread_sync stood between the wait and the store.  What the
// all-lanes form does differently is control flow: mbar_wait has two exits per lane (try_wait succeeded at once, or
// the out-of-line slow path returned), lanes take them at different times, and everything after them -- including the
// inline-asm store -- is reached through per-lane branches.  A ".sync.aligned" instruction must be executed by all
// lanes of the warp as ONE instruction; inline asm is not marked convergent for the compiler, so it may legally be
// cloned into both exits, and lanes arriving from different exits then run different copies of the store.  A
// __syncwarp or a vote between the wait and the store synchronises the lanes in time but does not undo such cloning,
// which fits the observation that neither cured it.  Whether that is the whole cause could not be confirmed (machine
// code is not inspected here, and the failing form is not run again); the single-poller form removes the per-lane
// branches from the path altogether -- the store is reached by straight-line code behind a shuffle -- and has not
// failed; tests/test_gemm_gpu.py repeats a full-size call twelve times and compares bit for bit.
__device__ __forceinline__ bool mbar_wait_warp(uint64_t* bar, uint32_t parity, int* abort_flag, unsigned* err) {
    int got = 1;
    if ((threadIdx.x & 31) == 0) got = mbar_wait(bar, parity, abort_flag, err) ? 1 : 0;
    got = __shfl_sync(0xffffffffu, got, 0);
    __syncwarp();
    return got != 0;
}

// Whole-warp wait for two or three barriers (mbar_wait_warp above with one poller and one broadcast for all: a
// wait for a barrier that is complete already costs about 150 cycles, most of them around the poll).
__device__ __forceinline__ bool mbar_wait_both(uint64_t* b0, uint32_t p0, uint64_t* b1, uint32_t p1, int* abort_flag, unsigned* err) {
    int got = 1;
    if ((threadIdx.x & 31) == 0) got = mbar_wait(b0, p0, abort_flag, err) && mbar_wait(b1, p1, abort_flag, err) ? 1 : 0;
    got = __shfl_sync(0xffffffffu, got, 0);
    __syncwarp();
    return got != 0;
}
__device__ __forceinline__ bool mbar_wait_three(uint64_t* b0, uint32_t p0, uint64_t* b1, uint32_t p1, uint64_t* b2, uint32_t p2, int* abort_flag, unsigned* err) {
    int got = 1;
    if ((threadIdx.x & 31) == 0)
        got = mbar_wait(b0, p0, abort_flag, err) && mbar_wait(b1, p1, abort_flag, err) && mbar_wait(b2, p2, abort_flag, err) ? 1 : 0;
    got = __shfl_sync(0xffffffffu, got, 0);
    __syncwarp();
    return got != 0;
}

// one lane of a converged warp
__device__ __forceinline__ bool elect_one() {
    uint32_t p;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(p));
    return p != 0;
}

__device__ __forceinline__ void tma_load_2d(void* dst, const CUtensorMap* map, uint64_t* bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(map)), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
        : "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

__device__ __forceinline__ void tc_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar)) : "memory");
}

// D[tmem] (+)= A[tmem] . B[smem descriptor]^T, M = 128, K = 16.
__device__ __forceinline__ void tc_mma_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t b_desc, uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}"
        ::"r"(d_tmem), "r"(a_tmem), "l"(b_desc), "r"(idesc), "r"(accumulate)
        : "memory");
}

__device__ __forceinline__ void tc_st32(uint32_t taddr, const uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16, "
        "%17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31, %32};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15]), "r"(v[16]), "r"(v[17]),
        "r"(v[18]), "r"(v[19]), "r"(v[20]), "r"(v[21]), "r"(v[22]), "r"(v[23]), "r"(v[24]), "r"(v[25]), "r"(v[26]),
        "r"(v[27]), "r"(v[28]), "r"(v[29]), "r"(v[30]), "r"(v[31])
        : "memory");
}

__device__ __forceinline__ void tc_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], "
        "{%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};"
        ::"r"(taddr), "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]),
        "r"(v[9]), "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

__device__ __forceinline__ void tc_ld32(uint32_t taddr, uint32_t (&v)[32]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]), "=r"(v[8]),
          "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15]), "=r"(v[16]),
          "=r"(v[17]), "=r"(v[18]), "=r"(v[19]), "=r"(v[20]), "=r"(v[21]), "=r"(v[22]), "=r"(v[23]), "=r"(v[24]),
          "=r"(v[25]), "=r"(v[26]), "=r"(v[27]), "=r"(v[28]), "=r"(v[29]), "=r"(v[30]), "=r"(v[31])
        : "r"(taddr)
        : "memory");
}


// Plain bulk copy global -> shared (no tensor map): both addresses 16-byte aligned, size a multiple of 16.
__device__ __forceinline__ void bulk_load(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    asm volatile(
        "cp.async.bulk.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1], %2, [%3];"
        ::"r"(smem_u32(dst)), "l"(reinterpret_cast<uint64_t>(src)), "r"(bytes), "r"(smem_u32(bar))
        : "memory");
}

}  // namespace mlxq
