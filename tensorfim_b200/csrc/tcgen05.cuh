// tcgen05.mma kind::mxf4 on bits expanded to 4-bit values: the pieces that the wave counter
// (count_f4.cu) and the packed family counter (count_pk.cu) share.
#pragma once

#include "tfim_internal.h"

namespace tfim {
namespace {

constexpr uint32_t kMbarSpin = 1u << 22;   // try_wait attempts before a wait gives up

__device__ __forceinline__ uint32_t smem_u32(const void* p) { return (uint32_t)__cvta_generic_to_shared(p); }

__device__ __forceinline__ void st_shared_v4(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}

// K-major, 128-byte swizzle shared-memory matrix descriptor: start address, leading byte
// offset 16 (unused by swizzled K-major layouts), stride byte offset 1024 (8-row groups),
// version 1, layout SWIZZLE_128B.
__device__ __forceinline__ uint64_t smem_desc(uint32_t addr) {
    uint64_t d = 0;
    d |= (uint64_t)((addr >> 4) & 0x3FFF);
    d |= (uint64_t)1 << 16;
    d |= (uint64_t)(1024 >> 4) << 32;
    d |= (uint64_t)1 << 46;
    d |= (uint64_t)2 << 61;
    return d;
}

// Instruction descriptor of kind::mxf4: A and B e2m1 (format 1), both K-major, UE8M0 scales,
// scale ids 0, N columns, M = 128.
__device__ __forceinline__ uint32_t idesc_mxf4(int n) {
    return (1u << 7) | (1u << 10) | ((uint32_t)(n >> 3) << 17) | (1u << 23) | ((uint32_t)(128 >> 4) << 24);
}

__device__ __forceinline__ void mma_mxf4(uint32_t tmem_d, uint64_t da, uint64_t db, uint32_t idesc, uint32_t sf,
                                         uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], %1, %2, %3, [%4], [%4], p;\n\t"
        "}\n" ::"r"(tmem_d),
        "l"(da), "l"(db), "r"(idesc), "r"(sf), "r"(accumulate));
}

// The same with the A operand in tensor memory: lane = row, a 32-bit cell holds eight values.
__device__ __forceinline__ void mma_mxf4_ta(uint32_t tmem_d, uint32_t tmem_a, uint64_t db, uint32_t idesc, uint32_t sf,
                                            uint32_t accumulate) {
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "setp.ne.b32 p, %5, 0;\n\t"
        "tcgen05.mma.cta_group::1.kind::mxf4.block_scale.scale_vec::2X [%0], [%1], %2, %3, [%4], [%4], p;\n\t"
        "}\n" ::"r"(tmem_d),
        "r"(tmem_a), "l"(db), "r"(idesc), "r"(sf), "r"(accumulate));
}

__device__ __forceinline__ void mbar_init(uint32_t bar, uint32_t count) {
    asm volatile("mbarrier.init.shared::cta.b64 [%0], %1;" ::"r"(bar), "r"(count) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint32_t bar) {
    asm volatile("{\n\t.reg .b64 st;\n\tmbarrier.arrive.shared::cta.b64 st, [%0];\n\t}" ::"r"(bar) : "memory");
}
__device__ __forceinline__ bool mbar_try_wait(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t"
        ".reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t"
        "}\n"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
// Bounded wait on phase `parity`; false when the limit expired.
__device__ __forceinline__ bool mbar_wait(uint32_t bar, uint32_t parity) {
    for (uint32_t k = 0; k < kMbarSpin; k++)
        if (mbar_try_wait(bar, parity)) return true;
    return false;
}
__device__ __forceinline__ void tc_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}

// One value into 16 columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_fill16(uint32_t taddr, uint32_t v) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {"
        "%1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1, %1};" ::"r"(taddr),
        "r"(v)
        : "memory");
}
// 16 columns of this warp's 32 lanes.
__device__ __forceinline__ void tmem_st16(uint32_t taddr, const uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x16.b32 [%0], {"
        "%1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15, %16};" ::"r"(taddr),
        "r"(v[0]), "r"(v[1]), "r"(v[2]), "r"(v[3]), "r"(v[4]), "r"(v[5]), "r"(v[6]), "r"(v[7]), "r"(v[8]), "r"(v[9]),
        "r"(v[10]), "r"(v[11]), "r"(v[12]), "r"(v[13]), "r"(v[14]), "r"(v[15])
        : "memory");
}

// The accumulator's registers are written asynchronously by tcgen05.ld and are valid only
// after tcgen05.wait::ld; both sit in one asm statement, so nothing reads them in between.
__device__ __forceinline__ void tmem_ld16(uint32_t taddr, uint32_t (&v)[16]) {
    asm volatile(
        "tcgen05.ld.sync.aligned.32x32b.x16.b32 {"
        "%0, %1, %2, %3, %4, %5, %6, %7, %8, %9, %10, %11, %12, %13, %14, %15"
        "}, [%16];\n\t"
        "tcgen05.wait::ld.sync.aligned;"
        : "=r"(v[0]), "=r"(v[1]), "=r"(v[2]), "=r"(v[3]), "=r"(v[4]), "=r"(v[5]), "=r"(v[6]), "=r"(v[7]),
          "=r"(v[8]), "=r"(v[9]), "=r"(v[10]), "=r"(v[11]), "=r"(v[12]), "=r"(v[13]), "=r"(v[14]), "=r"(v[15])
        : "r"(taddr)
        : "memory");
}


// The three scale regions, kScaleCols columns each, of this warp's 32 lanes: every byte 2, 1 and 1/2
// (UE8M0), so that the regions do not depend on the scale factors' layout.
constexpr uint32_t kScaleCols = 16;
__device__ __forceinline__ void tmem_fill_scales(uint32_t lanes) {
    tmem_fill16(lanes, 0x80808080u);
    tmem_fill16(lanes + kScaleCols, 0x7F7F7F7Fu);
    tmem_fill16(lanes + 2 * kScaleCols, 0x7E7E7E7Eu);
    asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory");
}

__device__ __forceinline__ void tc_fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void tc_fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }

// Tensor-memory allocation by one warp (the address into shared memory), and its release.
__device__ __forceinline__ void tmem_alloc(uint32_t smem_addr, uint32_t cols) {
    asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem_addr), "r"(cols));
    asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;");
}
__device__ __forceinline__ void tmem_free(uint32_t tmem, uint32_t cols) {
    asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(cols));
}

// 128 bits of a row as the four 16-byte chunks c0, 2 + c0, 4 + c0, 6 + c0 of its 128-byte K block
// (swizzled by the row's place rx in its group of eight): chunk pair k holds the bits that nibble
// mask k picks, as the e2m1 values 0.5, 1, 2 and 2.
__device__ __forceinline__ void store_nibbles(uint32_t o, uint32_t c0, uint32_t rx, uint4 x) {
    st_shared_v4(o + (((0 + c0) ^ rx) << 4), x.x & 0x11111111u, x.y & 0x11111111u, x.z & 0x11111111u, x.w & 0x11111111u);
    st_shared_v4(o + (((2 + c0) ^ rx) << 4), x.x & 0x22222222u, x.y & 0x22222222u, x.z & 0x22222222u, x.w & 0x22222222u);
    st_shared_v4(o + (((4 + c0) ^ rx) << 4), x.x & 0x44444444u, x.y & 0x44444444u, x.z & 0x44444444u, x.w & 0x44444444u);
    st_shared_v4(o + (((6 + c0) ^ rx) << 4), (x.x >> 1) & 0x44444444u, (x.y >> 1) & 0x44444444u, (x.z >> 1) & 0x44444444u,
                 (x.w >> 1) & 0x44444444u);
}

}  // namespace
}  // namespace tfim
