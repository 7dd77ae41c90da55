// PTX pieces shared by the tcgen05 GEMM kernels: bounded mbarrier wait, operand descriptor, TMEM reads, TMA tile loads.
#pragma once
#include "q3_common.cuh"

namespace q3 {

constexpr int TC_BK = 64;          // k per stage: 64 bf16 = one 128-byte swizzle row
constexpr unsigned long long TC_WAIT_NS = 200ull * 1000 * 1000;

__device__ __forceinline__ uint32_t tc_smem(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }
__device__ __forceinline__ unsigned long long tc_ns() { unsigned long long t; asm volatile("mov.u64 %0, %%globaltimer;" : "=l"(t)); return t; }

// bounded mbarrier wait; on timeout sets *abort_flag and returns false
// PARK: the thread may sleep up to 20 us between two looks (it wakes when the phase completes).
template <bool PARK = false>
[[nodiscard]] __device__ __forceinline__ bool tc_wait(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t site,
                                                      unsigned long long limit = TC_WAIT_NS) {
    unsigned it = 0;
    unsigned long long t0 = 0;
    for (;;) {
        uint32_t ok;
        if constexpr (PARK)
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2, %3;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok) : "r"(tc_smem(bar)), "r"(parity), "r"(20000u) : "memory");
        else
            asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                         : "=r"(ok) : "r"(tc_smem(bar)), "r"(parity) : "memory");
        if (ok) return true;
        if (*abort_flag) return false;
        if ((++it & 63u) == 0) {
            const unsigned long long t = tc_ns();
            if (t0 == 0) t0 = t;
            else if (t - t0 > limit) {
                report(status, ST_MBAR_TIMEOUT, site, parity);
                *abort_flag = 1;
                return false;
            }
        }
    }
}

// The same for a whole converged warp: one lane polls.  32 polling lanes are 32 requests to the barrier unit, and those of the
// epilogue warps stand in front of the MMA thread's own (a wait that was already over took it 190 ns instead of 30).  It is
// parked: looks in quick succession cost 40 / 64 sequences 1330 / 2031 us a step, parked 1318 / 2022, a prompt of 512 tokens 1380 and 1370.
[[nodiscard]] __device__ __forceinline__ bool tc_wait_warp(uint64_t* bar, uint32_t parity, volatile int* abort_flag, uint32_t* status, uint32_t site,
                                                           unsigned long long limit = TC_WAIT_NS) {
    return one_lane_waits([&] { return tc_wait<true>(bar, parity, abort_flag, status, site, limit); });
}

// After a wait has given up: let what is still under way to this block land before its memory is somebody else's.  Bounded, reports nothing.
static __device__ __noinline__ void tc_drain(uint64_t* bar, uint32_t parity) {
    const unsigned long long t0 = tc_ns();
    uint32_t ok = 0;
    while (!ok && tc_ns() - t0 <= TC_WAIT_NS)
        asm volatile("{\n\t.reg .pred p;\n\tmbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\tselp.u32 %0, 1, 0, p;\n\t}"
                     : "=r"(ok) : "r"(tc_smem(bar)), "r"(parity) : "memory");
}

// shared-memory matrix descriptor of a K-major tile with 128-byte swizzle: rows of 128 bytes, 8-row
// groups 1024 bytes apart (stride byte offset), descriptor version 1 (Blackwell)
__device__ __forceinline__ uint64_t tc_desc(uint32_t smem_addr) {
    uint64_t d = 0;
    d |= (uint64_t)((smem_addr & 0x3ffffu) >> 4);        // start address, bits [0,14)
    d |= (uint64_t)1 << 16;                              // leading byte offset (unused with swizzle), bits [16,30)
    d |= (uint64_t)(1024 >> 4) << 32;                    // stride byte offset, bits [32,46)
    d |= (uint64_t)1 << 46;                              // version
    d |= (uint64_t)2 << 61;                              // SWIZZLE_128B
    return d;
}

__device__ __forceinline__ void tc_ld32(uint32_t (&r)[32], uint32_t taddr) {   // 32 columns of this warp's 32 TMEM lanes; no wait
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x32.b32 "
                 "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
                 "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
                   "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
                   "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
                 : "r"(taddr) : "memory");
}

__device__ __forceinline__ void tc_ld16(uint32_t* r, uint32_t taddr) {   // 16 columns of this warp's 32 TMEM lanes; no wait
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15}, [%16];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
                   "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
                 : "r"(taddr) : "memory");
}

__device__ __forceinline__ void tc_ld8(uint32_t* r, uint32_t taddr) {   // 8 columns of this warp's 32 TMEM lanes; no wait
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]) : "r"(taddr) : "memory");
}

__device__ __forceinline__ void tc_ld4(uint32_t (&r)[4], uint32_t taddr) {   // 4 columns of this warp's 32 TMEM lanes; no wait
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x4.b32 {%0, %1, %2, %3}, [%4];" : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]) : "r"(taddr) : "memory");
}

// one 2-D box [rows of the map's box] x [64 k] into shared memory, counted on an mbarrier
__device__ __forceinline__ void tc_load_box(uint32_t dst, const void* map, int k, int row, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];"
                 ::"r"(dst), "l"(map), "r"(k), "r"(row), "r"(tc_smem(bar)) : "memory");
}
// a 3-D box [all planes] x [rows of the map's box] x [64 k]
__device__ __forceinline__ void tc_load_planes(uint32_t dst, const void* map, int k, int row, uint64_t* bar) {
    asm volatile("cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];"
                 ::"r"(dst), "l"(map), "r"(k), "r"(row), "r"(0), "r"(tc_smem(bar)) : "memory");
}

}  // namespace q3
