// Blackwell (sm_100-family) building blocks in inline PTX: mbarriers, TMA
// tensor copies, TMEM allocation, tcgen05.mma (kind::f16, BF16 in, FP32
// accumulate in TMEM) and tcgen05.ld.  Every wait has a time limit: on
// timeout the waiter records an error in the kernel's error word and the
// kernel winds down (waits, bounded, for its own copies/MMAs, frees TMEM).
#pragma once

#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace synk {
namespace umma {

__device__ __forceinline__ uint32_t smem_u32(const void *p) { return (uint32_t)__cvta_generic_to_shared(p); }

// ---- mbarrier -------------------------------------------------------------------
__device__ __forceinline__ void mbar_init(uint64_t *bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(smem_u32(bar)), "r"(count) : "memory");
}
__device__ __forceinline__ void fence_mbar_init() {
    asm volatile("fence.mbarrier_init.release.cluster;" ::: "memory");
}
__device__ __forceinline__ void mbar_arrive_expect_tx(uint64_t *bar, uint32_t bytes) {
    asm volatile("mbarrier.arrive.expect_tx.shared::cta.b64 _, [%0], %1;" ::"r"(smem_u32(bar)), "r"(bytes)
                 : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint64_t *bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(smem_u32(bar)), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Time limits of the spin waits are counted in SM clock cycles (clock64, a
// register read) rather than %globaltimer, whose read is slow enough to
// delay every hand-off between the pipeline's warps.  2.2 cycles per ns is
// above the maximum SM clock, so a limit of limit_ns lasts at least limit_ns.
__device__ __forceinline__ long long limit_cycles(unsigned long long limit_ns) {
    return (long long)(limit_ns * 11ull / 5ull);
}

// Waits for the phase of `parity`; false when the limit ran out or another
// thread of the kernel already failed (err != 0).  On timeout err is set.
// The error word (a global load) is only polled once a wait has lasted about
// 100 us, so healthy hand-offs never touch it.
__device__ __forceinline__ bool mbar_wait(uint64_t *bar, uint32_t parity, int *err, unsigned long long limit_ns) {
    if (mbar_try_wait(bar, parity)) return true;
    const long long c0 = clock64();
    const long long lim = limit_cycles(limit_ns);
    for (uint32_t i = 1;; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 1023u) == 0u) {
            const long long dc = clock64() - c0;
            if (dc > 220000ll && *(volatile int *)err) return false;
            if (dc > lim || i > (1u << 30)) {
                atomicExch(err, 3);   // SYNK_ETIMEOUT
                return false;
            }
        }
    }
}

// Wind-down wait for work this thread itself started (copies or MMAs in
// flight): ignores other threads' failures, gives up after limit_ns.
__device__ __forceinline__ bool mbar_drain(uint64_t *bar, uint32_t parity, unsigned long long limit_ns) {
    const long long c0 = clock64();
    const long long lim = limit_cycles(limit_ns);
    for (uint32_t i = 0;; ++i) {
        if (mbar_try_wait(bar, parity)) return true;
        if ((i & 1023u) == 1023u && (clock64() - c0 > lim || i > (1u << 30))) return false;
    }
}

// ---- TMA (tensor copies global -> shared, completion on an mbarrier) --------------
__device__ __forceinline__ void tma_load_2d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1)
        : "memory");
}
__device__ __forceinline__ void tma_load_3d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1, int c2) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5}], [%2];" ::"r"(
            smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2)
        : "memory");
}
__device__ __forceinline__ void tma_load_4d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1, int c2,
                                            int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6}], "
        "[%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
__device__ __forceinline__ void tma_load_5d(void *dst, const CUtensorMap *map, uint64_t *bar, int c0, int c1, int c2,
                                            int c3, int c4) {
    asm volatile(
        "cp.async.bulk.tensor.5d.shared::cluster.global.mbarrier::complete_tx::bytes [%0], [%1, {%3, %4, %5, %6, "
        "%7}], [%2];" ::"r"(smem_u32(dst)),
        "l"(map), "r"(smem_u32(bar)), "r"(c0), "r"(c1), "r"(c2), "r"(c3), "r"(c4)
        : "memory");
}
// Shared -> global, completion by bulk group of the issuing thread.
__device__ __forceinline__ void tma_store_4d(const CUtensorMap *map, const void *src, int c0, int c1, int c2, int c3) {
    asm volatile(
        "cp.async.bulk.tensor.4d.global.shared::cta.bulk_group [%0, {%2, %3, %4, %5}], [%1];" ::"l"(map),
        "r"(smem_u32(src)), "r"(c0), "r"(c1), "r"(c2), "r"(c3)
        : "memory");
}
__device__ __forceinline__ void bulk_commit() { asm volatile("cp.async.bulk.commit_group;" ::: "memory"); }
// All but the newest KEEP groups of this thread have left shared memory.
template <int KEEP>
__device__ __forceinline__ void bulk_wait_read() {
    asm volatile("cp.async.bulk.wait_group.read %0;" ::"n"(KEEP) : "memory");
}
__device__ __forceinline__ void bulk_wait_all() { asm volatile("cp.async.bulk.wait_group 0;" ::: "memory"); }
// Orders this thread's shared-memory writes before later copies of them.
__device__ __forceinline__ void fence_async_shared() {
    asm volatile("fence.proxy.async.shared::cta;" ::: "memory");
}
__device__ __forceinline__ void tma_prefetch_desc(const CUtensorMap *map) {
    asm volatile("prefetch.tensormap [%0];" ::"l"(map) : "memory");
}

// ---- TMEM ---------------------------------------------------------------------------
// Allocation by one full warp; the TMEM address is written to shared memory.
__device__ __forceinline__ void tmem_alloc(uint32_t *dst, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_u32(dst)), "r"(ncols)
                 : "memory");
}
__device__ __forceinline__ void tmem_relinquish() {
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}
__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// ---- descriptors ----------------------------------------------------------------------
// Shared-memory matrix descriptor of a K-major operand tile in the canonical
// swizzled layout written by TMA: rows of `row_bytes` (64 or 128) with the
// 16-byte chunks of row r XOR-permuted by r%8, 8-row groups `8*row_bytes`
// apart.  Fields: start address >> 4 (bits 0-13), leading-dimension offset
// (bits 16-29, unused for swizzled K-major, 1), stride-dimension offset >> 4
// (bits 32-45), the fixed value 1 in bits 46-48, swizzle mode in bits 61-63
// (2 = 128-byte, 4 = 64-byte).  Low half: the address and the leading-dimension
// offset; high half: a constant of the layout.
// A 128-byte-swizzled view may start r rows into a TMA-written tile: the XOR
// pattern is taken from the absolute shared-memory address, as TMA writes it,
// so the view needs no base offset.
__device__ __forceinline__ uint32_t smem_desc_lo(uint32_t saddr) { return ((saddr & 0x3FFFFu) >> 4) | 0x10000u; }
__device__ __forceinline__ uint32_t smem_desc_hi(uint32_t row_bytes) {
    return ((8u * row_bytes) >> 4) | (1u << 14) | ((row_bytes == 128u ? 2u : 4u) << 29);
}
// Instruction descriptor of tcgen05.mma kind::f16: D = F32 (bits 4-5 = 1),
// A = B = BF16 (bits 7-9 = 1, 10-12 = 1), both K-major (bits 15, 16 = 0),
// N >> 3 in bits 17-22, M >> 4 in bits 24-28.
__host__ __device__ constexpr uint32_t idesc_bf16(int M, int N) {
    return (1u << 4) | (1u << 7) | (1u << 10) | ((uint32_t)(N >> 3) << 17) | ((uint32_t)(M >> 4) << 24);
}

// ---- MMA ----------------------------------------------------------------------------------
// Descriptors as 32-bit halves: the low one moves from step to step (the start
// address >> 4), the high one is a constant.
__device__ __forceinline__ void mma_bf16(uint32_t d_tmem, uint32_t alo, uint32_t ahi, uint32_t blo, uint32_t bhi,
                                         uint32_t idesc, uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t.reg .b64 da, db;\n\t"
        "mov.b64 da, {%1, %2};\n\t"
        "mov.b64 db, {%3, %4};\n\t"
        "setp.ne.b32 p, %6, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::f16 [%0], da, db, %5, p;\n\t}" ::"r"(d_tmem),
        "r"(alo), "r"(ahi), "r"(blo), "r"(bhi), "r"(idesc), "r"(accumulate)
        : "memory");
}
// One lane of a converged warp (always the same one), which the compiler knows
// to be a single lane, unlike `lane == 0`: tensor instructions issued under it
// measured 1.5 to 3 times as many per second.
__device__ __forceinline__ bool elect_one() {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok));
    return ok != 0;
}
// KS K steps of one chunk (one row span): descriptors advance by 32 bytes a
// step; `acc` false overwrites the accumulator at the first one.
template <int KS>
__device__ __forceinline__ void mma_steps(uint32_t dt, uint32_t al, uint32_t bl, uint32_t hi, uint32_t idesc, bool acc) {
#pragma unroll
    for (uint32_t kk = 0; kk < (uint32_t)KS; ++kk)
        mma_bf16(dt, al + 2u * kk, hi, bl + 2u * kk, hi, idesc, kk != 0u || acc ? 1u : 0u);
}
// The three taps of one strip with rows of ROW bytes: tap kx starts kx rows
// into the strip and kx * tap16 * 16 bytes further into the weights; 4 or 2 K steps.
template <int ROW>
__device__ __forceinline__ void mma_taps(bool four, uint32_t dt, uint32_t al, uint32_t bl, uint32_t tap16, uint32_t hi,
                                         uint32_t idesc, bool acc) {
    constexpr uint32_t kRow16 = ROW / 16;
    if (ROW == 128 && four) {
#pragma unroll
        for (uint32_t kx = 0; kx < 3u; ++kx)
            mma_steps<4>(dt, al + kRow16 * kx, bl + kx * tap16, hi, idesc, kx != 0u || acc);
    } else {
#pragma unroll
        for (uint32_t kx = 0; kx < 3u; ++kx)
            mma_steps<2>(dt, al + kRow16 * kx, bl + kx * tap16, hi, idesc, kx != 0u || acc);
    }
}
// Arrives on `bar` once every MMA issued so far by this thread has completed.
__device__ __forceinline__ void mma_commit(uint64_t *bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_u32(bar))
                 : "memory");
}

// 32 lanes x 32 consecutive 32-bit columns: thread t of the warp gets lane
// (taddr.lane + t), columns taddr.col .. +31.
__device__ __forceinline__ void tmem_ld_32x32(uint32_t taddr, float (&v)[32]) {
    uint32_t r[32];
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x32.b32 "
        "{%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, "
        "%16, %17, %18, %19, %20, %21, %22, %23, %24, %25, %26, %27, %28, %29, %30, %31}, [%32];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15]),
          "=r"(r[16]), "=r"(r[17]), "=r"(r[18]), "=r"(r[19]), "=r"(r[20]), "=r"(r[21]), "=r"(r[22]), "=r"(r[23]),
          "=r"(r[24]), "=r"(r[25]), "=r"(r[26]), "=r"(r[27]), "=r"(r[28]), "=r"(r[29]), "=r"(r[30]), "=r"(r[31])
        : "r"(taddr)
        : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 32; ++i) v[i] = __uint_as_float(r[i]);
}

// The same for 8 columns.
__device__ __forceinline__ void tmem_ld_32x8(uint32_t taddr, float (&v)[8]) {
    uint32_t r[8];
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0, %1, %2, %3, %4, %5, %6, %7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 8; ++i) v[i] = __uint_as_float(r[i]);
}

}  // namespace umma
}  // namespace synk
