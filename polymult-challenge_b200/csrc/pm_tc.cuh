// pm_tc.cuh -- tcgen05 (tensor core, kind::i8) and tensor-memory helpers shared by the byte-sliced
// GEMM kernels: TMEM allocation, MMA issue, TMEM loads and stores, descriptors, async copies.
#pragma once

#include "pm_async.cuh"
#include "pm_kernels.cuh"

namespace pm {
namespace {

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// whole warp
__device__ __forceinline__ void tmem_alloc(uint32_t* slot, uint32_t ncols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr(slot)),
                 "r"(ncols)
                 : "memory");
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
}
__device__ __forceinline__ void tmem_dealloc(uint32_t taddr, uint32_t ncols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(taddr), "r"(ncols) : "memory");
}

// One lane of a converged warp.
__device__ __forceinline__ uint32_t elect_one() {
    uint32_t e;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "elect.sync _|p, 0xffffffff;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(e));
    return e;
}

// D[tmem] (+)= A[smem] * B[smem]^T, unsigned bytes, s32 accumulate, issued by the lane with `mine`
// set and called by a whole converged warp: the loop around it then is
// warp-uniform and its descriptors stay in uniform registers.  Issued from a branch of one lane an
// MMA took ~80 clocks of descriptor moves (k_crt16, k_dec16), more than it runs at N <= 128.
__device__ __forceinline__ void umma_u8_if(uint32_t mine, uint32_t d_tmem, uint64_t adesc, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p, q;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "setp.ne.b32 q, %5, 0;\n\t"
        "@q tcgen05.mma.cta_group::1.kind::i8 [%0], %1, %2, %3, p;\n\t}" ::"r"(d_tmem),
        "l"(adesc), "l"(bdesc), "r"(idesc), "r"(accumulate), "r"(mine)
        : "memory");
}

// D[tmem] (+)= A[tmem] * B[smem]^T, unsigned bytes, s32 accumulate; one thread.  A in tensor
// memory is K-major: lane m holds row m, and each 32-bit column holds 4 consecutive K bytes.
__device__ __forceinline__ void umma_u8_ts(uint32_t d_tmem, uint32_t a_tmem, uint64_t bdesc, uint32_t idesc,
                                           uint32_t accumulate) {
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "setp.ne.b32 p, %4, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::i8 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d_tmem),
        "r"(a_tmem), "l"(bdesc), "r"(idesc), "r"(accumulate)
        : "memory");
}

// This warp's 32 TMEM lanes x 8 consecutive 32-bit columns from registers (asynchronous: visible
// to the tensor core after tmem_wait_st and a before-thread-sync fence).
__device__ __forceinline__ void tmem_st8(uint32_t taddr, const uint32_t (&r)[8]) {
    asm volatile("tcgen05.st.sync.aligned.32x32b.x8.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8};" ::"r"(taddr), "r"(r[0]),
                 "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7])
                 : "memory");
}
__device__ __forceinline__ void tmem_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }

// 16-byte asynchronous global -> shared copy, L2 only (both addresses 16-byte aligned)
__device__ __forceinline__ void cp_async16(void* dst, const void* src) {
    asm volatile("cp.async.cg.shared.global [%0], [%1], 16;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}

__device__ __forceinline__ void umma_commit(uint64_t* bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(smem_addr(bar))
                 : "memory");
}

// 32 TMEM lanes (this warp's) x 8 consecutive 32-bit columns, without waiting (as the 16-column form)
__device__ __forceinline__ void tmem_ld8_async(uint32_t taddr, uint32_t (&r)[8]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x8.b32 {%0,%1,%2,%3,%4,%5,%6,%7}, [%8];"
                 : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7])
                 : "r"(taddr)
                 : "memory");
}

// Waits for the warp's TMEM loads: four 8-column loads' registers
__device__ __forceinline__ void tmem_wait_ld_4x8(uint32_t (&a)[8], uint32_t (&b)[8], uint32_t (&c)[8], uint32_t (&d)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                   "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7]),
                   "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3]), "+r"(c[4]), "+r"(c[5]), "+r"(c[6]), "+r"(c[7]),
                   "+r"(d[0]), "+r"(d[1]), "+r"(d[2]), "+r"(d[3]), "+r"(d[4]), "+r"(d[5]), "+r"(d[6]), "+r"(d[7])
                 :
                 : "memory");
}

// 32 TMEM lanes (this warp's) x 16 consecutive 32-bit columns, without waiting: the registers
// are valid after a wait that names them (tmem_wait_ld_*): until then they may be neither read nor
// copied, and only the wait's operands keep the compiler from doing so.  Issuing several before one
// wait overlaps their latency.
__device__ __forceinline__ void tmem_ld16_async(uint32_t taddr, uint32_t (&r)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
        : "=r"(r[0]), "=r"(r[1]), "=r"(r[2]), "=r"(r[3]), "=r"(r[4]), "=r"(r[5]), "=r"(r[6]), "=r"(r[7]),
          "=r"(r[8]), "=r"(r[9]), "=r"(r[10]), "=r"(r[11]), "=r"(r[12]), "=r"(r[13]), "=r"(r[14]), "=r"(r[15])
        : "r"(taddr)
        : "memory");
}

// one 8-column load's registers
__device__ __forceinline__ void tmem_wait_ld_8(uint32_t (&a)[8]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7])
                 :
                 : "memory");
}

// one 16-column load's registers
__device__ __forceinline__ void tmem_wait_ld_16(uint32_t (&a)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                   "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15])
                 :
                 : "memory");
}

// two 16-column loads' registers (where the second was not issued, its values pass through)
__device__ __forceinline__ void tmem_wait_ld_2x16(uint32_t (&a)[16], uint32_t (&b)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;"
                 : "+r"(a[0]), "+r"(a[1]), "+r"(a[2]), "+r"(a[3]), "+r"(a[4]), "+r"(a[5]), "+r"(a[6]), "+r"(a[7]),
                   "+r"(a[8]), "+r"(a[9]), "+r"(a[10]), "+r"(a[11]), "+r"(a[12]), "+r"(a[13]), "+r"(a[14]), "+r"(a[15]),
                   "+r"(b[0]), "+r"(b[1]), "+r"(b[2]), "+r"(b[3]), "+r"(b[4]), "+r"(b[5]), "+r"(b[6]), "+r"(b[7]),
                   "+r"(b[8]), "+r"(b[9]), "+r"(b[10]), "+r"(b[11]), "+r"(b[12]), "+r"(b[13]), "+r"(b[14]), "+r"(b[15])
                 :
                 : "memory");
}

// Shared-memory matrix descriptor, K-major, no swizzle (layout type 0), Blackwell version 1.
__device__ __forceinline__ uint64_t sdesc(uint32_t saddr, uint32_t lbo, uint32_t sbo) {
    return (uint64_t)((saddr >> 4) & 0x3FFFu) | ((uint64_t)((lbo >> 4) & 0x3FFFu) << 16) |
           ((uint64_t)((sbo >> 4) & 0x3FFFu) << 32) | (1ull << 46);
}

// Instruction descriptor, kind::i8: D = s32, A = B = u8, both K-major, M = 128.
__device__ __forceinline__ uint32_t idesc_u8(int n) {
    return (2u << 4) | ((uint32_t)(n >> 3) << 17) | ((uint32_t)(TC_M >> 4) << 24);
}

// Issues D[:, col0 : col0 + nn) = A * B[row0 : row0 + nn, :]^T into TMEM column col0.
// acc: the first MMA adds to the accumulator too (a further block of the K dimension).  Called by a
// whole converged warp, whose lane with `mine` set issues (umma_u8_if).
__device__ __forceinline__ void issue_gemm_rows(uint32_t mine, uint32_t tmem_col, uint32_t a_base, uint32_t b_base, int row0, int nn,
                                                int kbytes, bool acc = false) {
    const uint32_t sbo = 8u * (uint32_t)kbytes;
    const uint32_t idesc = idesc_u8(nn);
    uint64_t ad = sdesc(a_base, 128u, sbo), bd = sdesc(b_base + (uint32_t)(row0 >> 3) * sbo, 128u, sbo);
#pragma unroll 4
    for (int kk = 0; kk < kbytes / 32; ++kk, ad += 16, bd += 16)  // 256 bytes in 16-byte units
        umma_u8_if(mine, tmem_col, ad, bd, idesc, (kk > 0 || acc) ? 1u : 0u);
}

// 4-byte asynchronous global -> shared copy (no register staging); cp_async_wait_all waits for
// all of this thread's.
__device__ __forceinline__ void cp_async4(void* dst, const void* src) {
    asm volatile("cp.async.ca.shared.global [%0], [%1], 4;" ::"r"(smem_addr(dst)), "l"(src) : "memory");
}
__device__ __forceinline__ void cp_async_wait_all() { asm volatile("cp.async.wait_all;" ::: "memory"); }

// One thread: expect and issue a copy of `bytes` (multiple of 16) in pieces of <= 32 KB.
__device__ __forceinline__ void bulk_g2s_all(void* dst, const void* src, uint32_t bytes, uint64_t* bar) {
    mbar_arrive_expect_tx(bar, bytes);
    for (uint32_t off = 0; off < bytes; off += 32768u) {
        const uint32_t n = min(32768u, bytes - off);
        bulk_g2s(static_cast<unsigned char*>(dst) + off, static_cast<const unsigned char*>(src) + off, n, bar);
    }
}

// Registers per thread of the calling warpgroup (4 aligned warps, all of them executing it), within
// the total the block was launched with.
template <int N>
__device__ __forceinline__ void regs_inc() {
    asm volatile("setmaxnreg.inc.sync.aligned.u32 %0;" ::"n"(N));
}
template <int N>
__device__ __forceinline__ void regs_dec() {
    asm volatile("setmaxnreg.dec.sync.aligned.u32 %0;" ::"n"(N));
}

}  // namespace
}  // namespace pm
