// Device helpers of the one-column tensor-core kernels (matvec_tc.cu, matvec_expert.cu): shared-memory loads by 32-bit address,
// tiled TMA loads, mma.sync forms, bounded waits of the consumer loops.
#pragma once
#include "common.cuh"

#include <cuda.h>

namespace flb {

namespace {

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds32(uint32_t addr) {
    uint32_t v;
    asm volatile("ld.shared.u32 %0, [%1];" : "=r"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
    return v;
}
__device__ __forceinline__ void sts64(uint32_t addr, uint32_t a, uint32_t b) {
    asm volatile("st.shared.v2.u32 [%0], {%1, %2};" ::"r"(addr), "r"(a), "r"(b) : "memory");
}
__device__ __forceinline__ void sts128(uint32_t addr, uint32_t a, uint32_t b, uint32_t c, uint32_t d) {
    asm volatile("st.shared.v4.b32 [%0], {%1, %2, %3, %4};" ::"r"(addr), "r"(a), "r"(b), "r"(c), "r"(d) : "memory");
}
__device__ __forceinline__ void sts32(uint32_t addr, uint32_t a) {
    asm volatile("st.shared.b32 [%0], %1;" ::"r"(addr), "r"(a) : "memory");
}
__device__ __forceinline__ void mbar_arrive(uint64_t *bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(smem_u32(bar)) : "memory");
}
// Tiled TMA loads into shared memory (2-D: x counts 8-byte elements, a multiple of 2; 3-D: lines of 128 bytes).
__device__ __forceinline__ void tma_box2(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar))
        : "memory");
}
__device__ __forceinline__ void tma_box3(uint32_t dst, const CUtensorMap *map, uint32_t line, uint32_t row, uint64_t *bar) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3, %4}], [%5];" ::"r"(dst),
        "l"(map), "r"(0), "r"(line), "r"(row), "r"(smem_u32(bar))
        : "memory");
}
// The same with an L2 eviction policy for the lines the copy touches (the weights pass through L2 once).
__device__ __forceinline__ void tma_box2_hint(uint32_t dst, const CUtensorMap *map, uint32_t x, uint32_t y, uint64_t *bar, uint64_t pol) {
    asm volatile(
        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3}], [%4], %5;" ::"r"(dst),
        "l"(map), "r"(x), "r"(y), "r"(smem_u32(bar)), "l"(pol)
        : "memory");
}
__device__ __forceinline__ void tma_box3_hint(uint32_t dst, const CUtensorMap *map, uint32_t line, uint32_t row, uint64_t *bar, uint64_t pol) {
    asm volatile(
        "cp.async.bulk.tensor.3d.shared::cluster.global.tile.mbarrier::complete_tx::bytes.L2::cache_hint [%0], [%1, {%2, %3, %4}], [%5], %6;" ::"r"(dst),
        "l"(map), "r"(0), "r"(line), "r"(row), "r"(smem_u32(bar)), "l"(pol)
        : "memory");
}
__device__ __forceinline__ uint64_t l2_policy_evict_first() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_first.b64 %0, 1.0;" : "=l"(p));
    return p;
}
__device__ __forceinline__ uint64_t l2_policy_evict_last() {
    uint64_t p;
    asm volatile("createpolicy.fractional.L2::evict_last.b64 %0, 1.0;" : "=l"(p));
    return p;
}
// Read-only 16-byte load whose line is kept in L2 in preference to others (small tensors every launch reads again)
__device__ __forceinline__ float4 ldg_keep(const float4 *p, uint64_t pol) {
    float4 v;
    asm volatile("ld.global.nc.L2::cache_hint.v4.f32 {%0, %1, %2, %3}, [%4], %5;" : "=f"(v.x), "=f"(v.y), "=f"(v.z), "=f"(v.w) : "l"(p), "l"(pol));
    return v;
}
// All threads of the prologue (every warp but the producer) meet here.
__device__ __forceinline__ void prologue_barrier(uint32_t nthreads) {
    asm volatile("bar.sync 1, %0;" ::"r"(nthreads) : "memory");
}
// D(16x8, f32) += A(16x16, f16, row) * B(16x8, f16, col)
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// D(16x8, s32) += A(16x32, u8, row) * B(32x8, s8, col). Lane (g, t): a0 / a1 = rows g / g + 8, k-slots 4t..4t+3;
// a2 / a3 = the same rows, k-slots 16+4t..; b0 / b1 = column g, the same two k-slot runs; c as for the f16 form.
__device__ __forceinline__ void imma16832(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                          uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.u8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// Signed weights.
__device__ __forceinline__ void imma16832_ss(int (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0, uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k32.row.col.s32.s8.s8.s32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+r"(c[0]), "+r"(c[1]), "+r"(c[2]), "+r"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// (a & b) | c in one instruction; b and c are constants the compiler keeps in registers
__device__ __forceinline__ uint32_t and_or(uint32_t a, uint32_t b, uint32_t c) {
    uint32_t d;
    asm("lop3.b32 %0, %1, %2, %3, 0xEA;" : "=r"(d) : "r"(a), "r"(b), "r"(c));
    return d;
}
// h - off for both halves (exact: the operands are small integers)
__device__ __forceinline__ uint32_t hsub2_u32(uint32_t h, __half2 off) {
    const __half2 r = __hsub2(*reinterpret_cast<const __half2 *>(&h), off);
    return *reinterpret_cast<const uint32_t *>(&r);
}
// The common case of a wait: the phase is already complete. The bounded polling loop stays out of line.
__device__ __noinline__ bool mbar_wait_slow(uint64_t *bar, uint32_t parity, uint32_t *status) {
    return mbar_wait_bounded(bar, parity, status);
}
// The form the consumer loops use: no exit out of the loop. `dead` (warp-uniform) is set when a wait ran out;
// from then on the warp waits for nothing any more (its results are void, the status word says so) and the
// launch still ends.
__device__ __forceinline__ void mbar_wait_or_die(uint64_t *bar, uint32_t parity, uint32_t *status, bool &dead) {
    if (dead || mbar_try_wait(bar, parity)) return;
    dead = !mbar_wait_slow(bar, parity, status);
}
// byte K of w as a float without the conversion pipe (the byte under 0x4B000000 is 2^23 + byte)
template <int K>
__device__ __forceinline__ float u8f(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7650u | K)) - 8388608.0f;
}
__device__ __forceinline__ uint32_t word_of(const uint4 &v, int i) { return i == 0 ? v.x : i == 1 ? v.y : i == 2 ? v.z : v.w; }

// Byte offset o of a row as the stage holds it: as it is, or in the swizzled 128-byte lines (see kPitch4).
__device__ __forceinline__ uint32_t q4_row_off(uint32_t o, uint32_t g, bool swz) {
    return swz ? (o & ~127u) + ((((o >> 4) ^ (g + (o >> 7))) & 7u) << 4) : o;
}
// byte K of w, which holds s + 128, as the float s (the byte under 0x4B000000 is 2^23 + 128 + s)
template <int K>
__device__ __forceinline__ float s8f(uint32_t w) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + K)) - 8388736.f;
}

} // namespace

} // namespace flb
