// Several activation columns in one pass over Q4_K tensors on the Blackwell tensor cores: tcgen05.mma with the unpacked
// weights (A) and the results (D) in tensor memory, the activation (B) in shared memory. The same job as matvec_tc_nx.cu
// (Y[p][r] (+)= dot(W[r], X[p]), p < P <= 16; the STREAM_DOT semantics of Task::nx, include/fastllm/fastllm.h:87-96), whose
// tensor instructions bring every 16 x 16 weights into registers once per 4 tokens: the more tokens and the larger the tensor,
// the better this form (matmul_tm_takes).
//
// Unit of work: a step = 128 rows x one 256-column super-block. The steps of all tensors of a launch lie on one line, tile after
// tile; every CTA takes an equal, contiguous piece of it. A tile that is shared by several CTAs leaves one plane of partial sums
// per CTA (planes that a tile does not need are written as zeros), which the next activation conversion adds in order: results
// are reproducible run to run.
//
// Roles of a CTA (20 warps), all coupled by mbarriers:
//   unpack (2 x 4 warps)   : every other step each; thread = row: packed bytes -> f16, written to tensor memory (tcgen05.st 32x32b)
//   epilogue (2 x 4 warps) : every other step each; thread = row: D out of tensor memory, scales and mins, sum over the steps in
//                            f32; the second hands its sums to the first at the end of a tile, which writes the results
//   weights (1 thread)     : the packed bytes of a step, one TMA box of 128 rows x 144 bytes, into a ring of stages
//   activation (1 thread)  : the step's B operand (one bulk copy of the image that act_convert_nx_kernel built), same ring
//   tensor (1 warp)        : 16 instructions (M 128, N 2 x 8 or 2 x 16 tokens as (hi, lo), K 16) per step
// Every wait is bounded; a wait that runs out sets the status word and an abort flag all roles watch, the launch then drains,
// frees its tensor memory and returns.
//
// Arithmetic as in matvec_tc_nx.cu: (q - 8) sc as exact f16, activation of 22 bits per 256-column block, chains of four
// instructions (64 columns) from zero, added with rounding: tcgen05.mma truncates its running sum exactly as mma.sync does (bias of
// a chain of 4: -5.4e-8 of the result with either, of 16: -2.1e-7). The mins: 8 d sc - dmin m of a sub-block, rounded once, times
// the sub-block's f32 sum.
//
// What bounds it (B200): issue slots. A step takes 2600 warp instructions besides the polls (324 per 16 rows; matvec_tc_nx.cu 413 for 8
// tokens, 560 for 16), over four schedulers at 0.6 a cycle; the tensor pipe is 9 % busy (an instruction takes 15 cycles for N 16, 20
// for N 32, with A in tensor memory; 40 with A in shared memory), the weights arrive at 5.9 TB/s when nothing else is done.
// 28672 x 4096 with its conversion: 25.8 us for 8 tokens and 34.9 for 16 (matvec_tc_nx.cu: 28.3 and 40.5); 2 tokens 23.9 (23.4).
#include "common.cuh"
#include "kernels.h"

#include <algorithm>
#include <cstdlib>
#include <cstring>

namespace flb {

namespace {

constexpr uint32_t kRows = 128;
constexpr uint32_t kUnpackWarps = 8, kLoadWarp = 16, kTensorWarp = 17, kThreads = 20 * 32;   // the epilogue's from kUnpackWarps on
constexpr uint32_t kSmemLimit = 227 * 1024;
constexpr uint32_t kMaxSlots = 8, kComb = 1024;   // in front of the ring: barriers, then (kComb) the sums that one half of the epilogue hands to the other
__host__ __device__ constexpr uint32_t head_of(uint32_t T) { return kComb + kRows * T * 4; }
constexpr uint32_t kACol = 0, kABuf = 128, kDCol = 256, kTmemCols = 512;
constexpr uint32_t kPitch = 144;   // bytes of a row of a step: an odd multiple of 16, so that the row-per-thread reads do not collide

// A stage: the rows' bytes, then the step's activation (the operand's four tiles, sub-block sums, block scales, sums of squares).
template <int T> constexpr uint32_t kSlot = (kRows * kPitch + T * 1064 + 1023) & ~1023u;
template <int T> constexpr uint32_t kSlots = (kSmemLimit - head_of(T)) / kSlot<T> < kMaxSlots ? (kSmemLimit - head_of(T)) / kSlot<T> : kMaxSlots;

struct TmT {
    float *y;
    size_t part_stride;
    uint32_t rows, ystride, base;   // base: where the tensor starts on the line
};
struct TmArgs {
    CUtensorMap map[3];   // [rows][pitch / 8] 8-byte elements, box 128 rows x kPitch
    TmT t[3];
    uint32_t n, steps, nblk, P, parts, whole;   // whole: a CTA takes whole tiles only
    const uint8_t *xq;
    int accumulate, rms;
    float eps;
    uint32_t *status;
};

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
__device__ __forceinline__ bool bar_try(uint32_t bar, uint32_t parity) {
    uint32_t ok;
    asm volatile(
        "{\n\t.reg .pred p;\n\t"
        "mbarrier.try_wait.parity.shared::cta.b64 p, [%1], %2;\n\t"
        "selp.u32 %0, 1, 0, p;\n\t}"
        : "=r"(ok)
        : "r"(bar), "r"(parity)
        : "memory");
    return ok != 0;
}
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
}
__device__ __forceinline__ uint64_t *bar_at(uint32_t addr) { return reinterpret_cast<uint64_t *>(__cvta_shared_to_generic(addr)); }

// Waits of a whole warp (the answer is the same for all lanes) and of one thread: at most a second, and no longer once
// another role of the CTA has given up.
__device__ __forceinline__ bool warp_wait_slow(uint32_t bar, uint32_t parity, uint32_t *status, volatile uint32_t *abort_flag) {
    const uint64_t t0 = globaltimer_ns();
    for (;;) {
        for (int i = 0; i < 4; ++i)
            if (__all_sync(0xffffffffu, bar_try(bar, parity))) return true;
        const bool late = globaltimer_ns() - t0 > kDefaultWaitNs, stop = *abort_flag != 0;
        if (__any_sync(0xffffffffu, late || stop)) {
            if (!stop) { atomicCAS(status, ST_OK, ST_WAIT_TIMEOUT); *abort_flag = 1u; }
            return false;
        }
    }
}
__device__ __forceinline__ bool warp_wait(uint32_t bar, uint32_t parity, uint32_t *status, uint32_t *abort_flag) {
    return __all_sync(0xffffffffu, bar_try(bar, parity)) || warp_wait_slow(bar, parity, status, abort_flag);
}
__device__ __forceinline__ bool one_wait_slow(uint32_t bar, uint32_t parity, uint32_t *status, volatile uint32_t *abort_flag) {
    const uint64_t t0 = globaltimer_ns();
    for (;;) {
        for (int i = 0; i < 4; ++i)
            if (bar_try(bar, parity)) return true;
        if (*abort_flag) return false;
        if (globaltimer_ns() - t0 > kDefaultWaitNs) {
            atomicCAS(status, ST_OK, ST_WAIT_TIMEOUT);
            *abort_flag = 1u;
            return false;
        }
    }
}
__device__ __forceinline__ bool one_wait(uint32_t bar, uint32_t parity, uint32_t *status, uint32_t *abort_flag) {
    return bar_try(bar, parity) || one_wait_slow(bar, parity, status, abort_flag);
}

__device__ __forceinline__ void fence_before() { asm volatile("tcgen05.fence::before_thread_sync;" ::: "memory"); }
__device__ __forceinline__ void fence_after() { asm volatile("tcgen05.fence::after_thread_sync;" ::: "memory"); }
// 32 lanes x 32 columns: r[i] = column i of the thread's lane
__device__ __forceinline__ void tm_store32(uint32_t addr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.32x32b.x32.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
        "%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(addr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
        "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// columns c .. c + 15 of this thread's lane; the values may be used after tm_wait_ld
__device__ __forceinline__ void tm_load16(uint32_t addr, float (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]),
                   "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
                 : "r"(addr)
                 : "memory");
}
// waits for the loads in flight; names their values, so that nothing uses them earlier
__device__ __forceinline__ void tm_wait_ld(float (&a)[16], float (&b)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) asm volatile("" : "+f"(a[i]), "+f"(b[i]));
}
__device__ __forceinline__ void tm_wait_ld(float (&a)[16], float (&b)[16], float (&c)[16], float (&d)[16]) {
    asm volatile("tcgen05.wait::ld.sync.aligned;" ::: "memory");
#pragma unroll
    for (int i = 0; i < 16; ++i) asm volatile("" : "+f"(a[i]), "+f"(b[i]), "+f"(c[i]), "+f"(d[i]));
}
// Shared-memory matrix descriptor: K-major, 128-byte swizzle, 8-row groups 1024 bytes apart.
__device__ __forceinline__ uint64_t b_desc(uint32_t saddr) {
    return (uint64_t)((saddr & 0x3FFFFu) >> 4) | ((uint64_t)(1024u >> 4) << 32) | (1ull << 46) | (2ull << 61);
}
__device__ __forceinline__ void tm_mma(uint32_t d, uint32_t a, uint64_t b, uint32_t idesc, uint32_t accumulate) {
    asm volatile("{\n\t.reg .pred p;\n\tsetp.ne.b32 p, %4, 0;\n\ttcgen05.mma.cta_group::1.kind::f16 [%0], [%1], %2, %3, p;\n\t}" ::"r"(d), "r"(a),
                 "l"(b), "r"(idesc), "r"(accumulate)
                 : "memory");
}
__device__ __forceinline__ void tm_commit(uint32_t bar) {
    asm volatile("tcgen05.commit.cta_group::1.mbarrier::arrive::one.shared::cluster.b64 [%0];" ::"r"(bar) : "memory");
}
// One lane of the warp, the same one every time. The tensor warp runs as a whole and branches on this only around its
// instructions: their operands stay in uniform registers (with one thread in a branch of its own, moving them there took
// most of the 135 cycles that an instruction cost; the unit itself needs 45 for N up to 64).
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }
__device__ __forceinline__ uint32_t hfma2_u32(uint32_t h, __half2 m, __half2 c) { return as_u32(__hfma2(as_h2(h), m, c)); }
// byte k of w as a float
__device__ __forceinline__ float u8f(uint32_t w, int k) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + k)) - 8388608.f; }

// two f32 at once
struct F2 { uint64_t v; };
__device__ __forceinline__ F2 f2(float a, float b) { F2 r; asm("mov.b64 %0, {%1, %2};" : "=l"(r.v) : "f"(a), "f"(b)); return r; }
__device__ __forceinline__ F2 f2(float a) { return f2(a, a); }
__device__ __forceinline__ void unpair(F2 x, float &a, float &b) { asm("mov.b64 {%0, %1}, %2;" : "=f"(a), "=f"(b) : "l"(x.v)); }
__device__ __forceinline__ F2 operator+(F2 a, F2 b) { F2 r; asm("add.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 operator*(F2 a, F2 b) { F2 r; asm("mul.rn.f32x2 %0, %1, %2;" : "=l"(r.v) : "l"(a.v), "l"(b.v)); return r; }
__device__ __forceinline__ F2 fma2(F2 a, F2 b, F2 c) { F2 r; asm("fma.rn.f32x2 %0, %1, %2, %3;" : "=l"(r.v) : "l"(a.v), "l"(b.v), "l"(c.v)); return r; }
__device__ __forceinline__ void lds_f2x2(uint32_t addr, F2 &a, F2 &b) {
    asm volatile("ld.shared.v2.u64 {%0, %1}, [%2];" : "=l"(a.v), "=l"(b.v) : "r"(addr));
}

// ---- pieces: the runs of consecutive steps of one tile that this CTA owns --------------------------------------------
struct Piece { uint32_t ten, tile, b0, b1, plane; };
struct Walk { uint32_t pos, hi; };
__device__ __forceinline__ uint32_t share_lo(const TmArgs &a, uint32_t c) { return a.steps / gridDim.x * c + a.steps % gridDim.x * c / gridDim.x; }
__device__ __forceinline__ Walk walk_begin(const TmArgs &a) { return Walk{share_lo(a, blockIdx.x), share_lo(a, blockIdx.x + 1)}; }
__device__ __forceinline__ bool walk_next(const TmArgs &a, Walk &w, Piece &p) {
    if (a.whole) w.pos = (w.pos + a.nblk - 1) / a.nblk * a.nblk;   // (every tensor starts on a multiple)
    if (w.pos >= w.hi) return false;
    uint32_t j = 0;
    if (a.n > 1 && w.pos >= a.t[1].base) j = 1;
    if (a.n > 2 && w.pos >= a.t[2].base) j = 2;
    const uint32_t st = w.pos - a.t[j].base;
    p.ten = j; p.tile = st / a.nblk; p.b0 = st - p.tile * a.nblk;
    p.b1 = a.whole ? a.nblk : min(a.nblk, p.b0 + w.hi - w.pos);
    p.plane = 0;   // = the CTAs in front that have steps of this tile
    if (p.b0) {
        p.plane = 1;
        while (share_lo(a, blockIdx.x - p.plane) > w.pos - p.b0) ++p.plane;
    }
    w.pos += p.b1 - p.b0;
    return true;
}

// Offsets in shared memory.
constexpr uint32_t kRawFull = 0, kActFull = kRawFull + 8 * kMaxSlots, kEmpty = kActFull + 8 * kMaxSlots, kAFull = kEmpty + 8 * kMaxSlots,
                   kAEmpty = kAFull + 16, kDFull = kAEmpty + 16, kDEmpty = kDFull + 32, kCombFull = kDEmpty + 32, kCombEmpty = kCombFull + 32,
                   kDrain = kCombEmpty + 32, kTmemPtr = kDrain + 8,
                   kAbort = kTmemPtr + 4;
static_assert(kAbort + 4 <= kComb, "head");

// ---- unpack: the weights of a warp's 32 rows as f16 into 128 columns of tensor memory ----------------------------------
// Thread = row (address r). A masked nibble is the subnormal f16 q 2^-24 (q 2^-20 in the
// high nibble), one FMA makes it (q - 8) sc 2^-14, exact. Column 32 c + 4 w + {0, 1, 2, 3}: word w of chunk c, low nibbles of
// bytes (0, 2), of bytes (1, 3), high nibbles of the same.
__device__ __forceinline__ void unpack_q4k(uint32_t r, uint32_t tm) {
    const uint4 hd = lds128(r);
    // 6-bit scales (packing: fl_q4k_scale_min, src/runtime/quants.h:121-129)
    const uint32_t sc_lo = hd.y & 0x3F3F3F3Fu, sc_hi = (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u);
    const __half2 k1024 = __floats2half2_rn(1024.f, 1024.f), k64 = __floats2half2_rn(64.f, 64.f);
    const __half2 km8 = __floats2half2_rn(-0.00048828125f, -0.00048828125f);   // -8 2^-14
    const uint32_t ML = 0x000F000Fu, MH = 0x00F000F0u;
#pragma unroll 1
    for (uint32_t c = 0; c < 4; ++c) {   // (rolled: the roles of a CTA share the instruction caches)
        const uint4 wa = lds128(r + 16 + 32 * c), wb = lds128(r + 32 + 32 * c);
        const uint32_t sc = (c & 2u ? sc_hi : sc_lo) >> (16u * (c & 1u));
        const __half2 s0 = __hsub2(as_h2(__byte_perm(sc, 0x64646464u, 0x4040u)), k1024), s1 = __hsub2(as_h2(__byte_perm(sc, 0x64646464u, 0x4141u)), k1024);
        const __half2 sL = __hmul2(s0, k1024), kL = __hmul2(s0, km8), sH = __hmul2(s1, k64), kH = __hmul2(s1, km8);
        uint32_t o[32];
#pragma unroll
        for (int j = 0; j < 8; ++j) {
            const uint4 &q = j < 4 ? wa : wb;
            const uint32_t W = (j & 3) == 0 ? q.x : (j & 3) == 1 ? q.y : (j & 3) == 2 ? q.z : q.w, V = W >> 8;
            o[4 * j] = hfma2_u32(W & ML, sL, kL);
            o[4 * j + 1] = hfma2_u32(V & ML, sL, kL);
            o[4 * j + 2] = hfma2_u32(W & MH, sH, kH);
            o[4 * j + 3] = hfma2_u32(V & MH, sH, kH);
        }
        tm_store32(tm + 32 * c, o);
    }
}
// ---- epilogue of one step: acc[i] += the step's results of tokens 2 i, 2 i + 1 -----------------------------------------
// The four results of a step (D: 4 x N columns; N = 2 NT: hi columns of the tokens, then lo columns).
struct Ring { uint32_t slot, par; };
struct Epi {
    uint32_t smem, tmem;   // tmem: this warp's lanes
    uint32_t *status, *abort_flag;
};
// Each half of the epilogue has R / 2 of the D buffers for itself.
template <int NT, int R, typename F>
__device__ __forceinline__ bool step_results(const Epi &e, Ring &d, uint32_t lane, F &&use) {
    if (!warp_wait(e.smem + kDFull + 8 * d.slot, d.par, e.status, e.abort_flag)) return false;
    fence_after();
    const uint32_t at = e.tmem + kDCol + d.slot * (256 / R);
    float r0[16], r1[16], r2[16], r3[16];
    if constexpr (NT == 8) {   // (hi, lo) of the 8 tokens of each result
        tm_load16(at, r0); tm_load16(at + 16, r1); tm_load16(at + 32, r2); tm_load16(at + 48, r3);
        tm_wait_ld(r0, r1, r2, r3);
    } else {                   // two results at a time: r0, r1 hi and lo of one, r2, r3 of the other
        tm_load16(at, r0); tm_load16(at + 16, r1);
        tm_wait_ld(r0, r1);
        tm_load16(at + 32, r2); tm_load16(at + 48, r3);
        use(0, r0, r1);
        tm_wait_ld(r2, r3);
        tm_load16(at + 64, r0); tm_load16(at + 80, r1);
        use(1, r2, r3);
        tm_wait_ld(r0, r1);
        tm_load16(at + 96, r2); tm_load16(at + 112, r3);
        use(2, r0, r1);
        tm_wait_ld(r2, r3);
    }
    fence_before();
    __syncwarp();
    if (lane == 0) bar_arrive(e.smem + kDEmpty + 8 * d.slot);
    if constexpr (NT == 8) use(r0, r1, r2, r3);
    else use(3, r2, r3);
    if (R == 2) d.par ^= 1u;
    else if ((++d.slot & 1u) == 0) { d.slot -= 2; d.par ^= 1u; }
    return true;
}
template <int NT, int R>
__device__ __forceinline__ bool epi_step(const Epi &e, Ring &d, uint32_t lane, uint32_t row_addr, uint32_t side, F2 (&acc)[NT / 2]) {
    const uint32_t xs = side + NT * 32;
    F2 sum[NT / 2];
    const uint4 hd = lds128(row_addr);
    const float d8 = 8.f * h2f_bits((uint16_t)(hd.x & 0xFFFFu)), em = h2f_bits((uint16_t)(hd.x >> 16));
    const uint32_t sc[2] = {hd.y & 0x3F3F3F3Fu, (hd.w & 0x0F0F0F0Fu) | ((hd.y >> 2) & 0x30303030u)};
    const uint32_t mn[2] = {hd.z & 0x3F3F3F3Fu, ((hd.w >> 4) & 0x0F0F0F0Fu) | ((hd.z >> 2) & 0x30303030u)};
    // 8 d sc - dmin m of a sub-block, rounded once (both products are exact), times the sum of its activation
    F2 v[NT / 2];
#pragma unroll
    for (int k = 0; k < 8; ++k) {
        const F2 c = f2(fmaf(d8, u8f(sc[k >> 2], k & 3), -(em * u8f(mn[k >> 2], k & 3))));
#pragma unroll
        for (int i = 0; i < NT / 2; i += 2) {
            F2 s0, s1;
            lds_f2x2(side + k * (NT * 4) + i * 8, s0, s1);
            v[i] = k ? fma2(c, s0, v[i]) : c * s0;
            v[i + 1] = k ? fma2(c, s1, v[i + 1]) : c * s1;
        }
    }
    const F2 dq = f2(2048.f * d8);   // 2^14 d
    const auto add8 = [&](float (&a)[16], float (&b)[16], float (&c)[16], float (&f)[16]) {
#pragma unroll
        for (int i = 0; i < 4; ++i)
            sum[i] = ((f2(a[2 * i], a[2 * i + 1]) + f2(b[2 * i], b[2 * i + 1])) + (f2(c[2 * i], c[2 * i + 1]) + f2(f[2 * i], f[2 * i + 1]))) +
                     ((f2(a[8 + 2 * i], a[9 + 2 * i]) + f2(b[8 + 2 * i], b[9 + 2 * i])) + (f2(c[8 + 2 * i], c[9 + 2 * i]) + f2(f[8 + 2 * i], f[9 + 2 * i])));
    };
    const auto add16 = [&](int k, float (&h)[16], float (&l)[16]) {
#pragma unroll
        for (int i = 0; i < NT / 2; ++i) {
            const F2 s = f2(h[2 * i], h[2 * i + 1]) + f2(l[2 * i], l[2 * i + 1]);
            sum[i] = k ? sum[i] + s : s;
        }
    };
    if constexpr (NT == 8) { if (!step_results<NT, R>(e, d, lane, add8)) return false; }
    else { if (!step_results<NT, R>(e, d, lane, add16)) return false; }
#pragma unroll
    for (int i = 0; i < NT / 2; i += 2) {
        F2 x0, x1;
        lds_f2x2(xs + i * 8, x0, x1);
        acc[i] = fma2(x0, fma2(dq, sum[i], v[i]), acc[i]);
        acc[i + 1] = fma2(x1, fma2(dq, sum[i + 1], v[i + 1]), acc[i + 1]);
    }
    return true;
}

// The 16 instructions of a step (a: its weights, b: descriptor of its activation, dt: its four results).
template <int N>
__device__ __forceinline__ void tensor_step(uint32_t a, uint64_t b, uint32_t dt) {
    constexpr uint32_t idesc = (1u << 4) | ((N >> 3) << 17) | ((128u >> 4) << 24);   // f16 x f16 -> f32, K-major, M 128
#pragma unroll
    for (int m = 0; m < 16; ++m) tm_mma(dt + (m >> 2) * N, a + 8 * m, b + (uint64_t)((m >> 2) * N * 8 + (m & 3) * 2), idesc, m & 3);
}

template <int T>
__global__ void __launch_bounds__(kThreads, 1) matmul_tm_kernel(const __grid_constant__ TmArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr int R = T == 16 ? 2 : 4;   // D buffers (4 x N columns each)
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, smem = smem_u32(smem_raw);
    uint32_t *abort_flag = reinterpret_cast<uint32_t *>(smem_raw + kAbort);
    griddep_launch_dependents();
    if (tid == 0) {
        for (uint32_t i = 0; i < kMaxSlots; ++i) {
            mbar_init(bar_at(smem + kRawFull + 8 * i), 1);
            mbar_init(bar_at(smem + kActFull + 8 * i), 1);
            mbar_init(bar_at(smem + kEmpty + 8 * i), 4 + 4);   // the step's unpack warps and epilogue (which comes after the tensor core)
        }
        for (uint32_t i = 0; i < 2; ++i) { mbar_init(bar_at(smem + kAFull + 8 * i), 4); mbar_init(bar_at(smem + kAEmpty + 8 * i), 1); }
        for (uint32_t i = 0; i < (uint32_t)R; ++i) { mbar_init(bar_at(smem + kDFull + 8 * i), 1); mbar_init(bar_at(smem + kDEmpty + 8 * i), 4); }
        for (uint32_t i = 0; i < 4; ++i) { mbar_init(bar_at(smem + kCombFull + 8 * i), 1); mbar_init(bar_at(smem + kCombEmpty + 8 * i), 1); }
        mbar_init(bar_at(smem + kDrain), 1);
        *abort_flag = 0u;
        fence_barrier_init();
    }
    if (warp == kTensorWarp) {
        asm volatile("tcgen05.alloc.cta_group::1.sync.aligned.shared::cta.b32 [%0], %1;" ::"r"(smem + kTmemPtr), "r"(kTmemCols) : "memory");
        asm volatile("tcgen05.relinquish_alloc_permit.cta_group::1.sync.aligned;" ::: "memory");
    }
    fence_before();
    __syncthreads();
    fence_after();
    const uint32_t tmem = lds32(smem + kTmemPtr), stages = smem + head_of(T);
    Walk wk = walk_begin(a);
    Piece pc;
    Ring st{0, 0};   // the stage ring
    auto step_on = [&]() { if (++st.slot == kSlots<T>) { st.slot = 0; st.par ^= 1u; } };
    bool dead = false;
    // after an abort: waits for the copies in flight, those of the last n steps of the ring's barriers at `full`
    auto drain = [&](uint32_t full, uint32_t n) {
        for (uint32_t k = 0; dead && k < min(n, kSlots<T>); ++k) {
            const uint32_t i = n - 1 - k;
            const uint64_t t0 = globaltimer_ns();
            while (!bar_try(smem + full + 8 * (i % kSlots<T>), (i / kSlots<T>) & 1u) && globaltimer_ns() - t0 < kDefaultWaitNs) {}
        }
    };

    // 640 threads start with 96 registers each: 2 x 80 (unpack) + 2 x 128 (epilogue) + 64 = 5 x 96
    if (warp < kUnpackWarps) asm volatile("setmaxnreg.dec.sync.aligned.u32 80;");
    else if (warp < kLoadWarp) asm volatile("setmaxnreg.inc.sync.aligned.u32 128;");
    else asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");

    if (warp < kUnpackWarps) {
        const uint32_t wg = warp >> 2, quad = warp & 3u;
        uint32_t turn = 0, par = 1;   // a fresh barrier passes a wait on parity 1
        while (!dead && walk_next(a, wk, pc)) {
            for (uint32_t blk = pc.b0; blk < pc.b1; ++blk, turn ^= 1u) {
                if (turn != wg) { step_on(); continue; }
                const uint32_t raw = stages + st.slot * kSlot<T>;
                if (!warp_wait(smem + kRawFull + 8 * st.slot, st.par, a.status, abort_flag) ||
                    !warp_wait(smem + kAEmpty + 8 * wg, par, a.status, abort_flag)) { dead = true; break; }
                fence_after();
                unpack_q4k(raw + (quad * 32 + lane) * kPitch, tmem + ((quad * 32) << 16) + kACol + wg * kABuf);
                tm_wait_st();
                fence_before();
                __syncwarp();
                if (lane == 0) { bar_arrive(smem + kAFull + 8 * wg); bar_arrive(smem + kEmpty + 8 * st.slot); }
                par ^= 1u;
                step_on();
            }
        }
    } else if (warp < kLoadWarp) {
        // ---- epilogue ----
        const uint32_t quad = warp & 3u, row = quad * 32 + lane;
        const uint32_t half = (warp - kUnpackWarps) >> 2;
        const Epi e{smem, tmem + ((quad * 32) << 16), a.status, abort_flag};
        Ring d{half * (R / 2), 0};
        uint32_t turn = 0, comb_par = half;
        griddep_wait();   // y and the sums of squares come from the kernels before
        constexpr uint32_t xb = T * 1064u;
        float inv = 1.f;   // lane p: 1 / rms of token p
        if (a.rms) {
            const uint8_t *ss_at = a.xq + T * 1060u + (lane & (T - 1)) * 4u;
            float ss = 0.f;
#pragma unroll 8
            for (uint32_t b = 0; b < a.nblk; ++b) ss += __ldcg(reinterpret_cast<const float *>(ss_at + (size_t)b * xb));
            inv = 1.0f / sqrtf(ss / (float)(a.nblk * 256u) + a.eps);
        }
        while (!dead && walk_next(a, wk, pc)) {
            const TmT &t = a.t[pc.ten];
            F2 acc[T / 2];
#pragma unroll
            for (int i = 0; i < T / 2; ++i) acc[i] = f2(0.f);
            for (uint32_t blk = pc.b0; blk < pc.b1; ++blk) {
                const uint32_t raw = stages + st.slot * kSlot<T>, side = raw + kRows * kPitch + T * 1024u;
                if (turn++ % 2 != half) { step_on(); continue; }
                if (!warp_wait(smem + kRawFull + 8 * st.slot, st.par, a.status, abort_flag) ||
                    !warp_wait(smem + kActFull + 8 * st.slot, st.par, a.status, abort_flag) ||
                    !epi_step<T, R>(e, d, lane, raw + row * kPitch, side, acc)) { dead = true; break; }
                __syncwarp();
                if (lane == 0) bar_arrive(smem + kEmpty + 8 * st.slot);
                step_on();
            }
            if (dead) break;
            const uint32_t comb = smem + kComb + (quad * (T / 2) * 32 + lane) * 8;
            if (half) {
                if (!warp_wait(smem + kCombEmpty + 8 * quad, comb_par, a.status, abort_flag)) { dead = true; break; }
#pragma unroll
                for (int i = 0; i < T / 2; ++i) asm volatile("st.shared.u64 [%0], %1;" ::"r"(comb + i * 256), "l"(acc[i].v) : "memory");
                __syncwarp();
                if (lane == 0) bar_arrive(smem + kCombFull + 8 * quad);
                comb_par ^= 1u;
                continue;
            }
            if (!warp_wait(smem + kCombFull + 8 * quad, comb_par, a.status, abort_flag)) { dead = true; break; }
#pragma unroll
            for (int i = 0; i < T / 2; ++i) {
                F2 o;
                asm volatile("ld.shared.u64 %0, [%1];" : "=l"(o.v) : "r"(comb + i * 256));
                acc[i] = acc[i] + o;
            }
            __syncwarp();
            if (lane == 0) bar_arrive(smem + kCombEmpty + 8 * quad);
            comb_par ^= 1u;
            const uint32_t grow = pc.tile * kRows + row;
            const bool in = grow < t.rows;
            float *plane = t.y + pc.plane * t.part_stride + grow;
            const uint32_t planes = pc.b1 == a.nblk ? a.parts : pc.plane + 1;   // the last CTA of a tile clears the planes the tile has no sums for
#pragma unroll
            for (int i = 0; i < T / 2; ++i) {
                float v[2];
                unpair(acc[i], v[0], v[1]);
#pragma unroll
                for (int k = 0; k < 2; ++k) {
                    const uint32_t p = 2 * i + k;
                    const float s = __shfl_sync(0xffffffffu, inv, p);
                    if (p >= a.P || !in) continue;
                    float *dst = plane + (size_t)p * t.ystride;
                    const float r = a.rms ? v[k] * s : v[k];
                    *dst = a.accumulate ? *dst + r : r;
#pragma unroll 1
                    for (uint32_t q = pc.plane + 1; q < planes; ++q) dst[(size_t)(q - pc.plane) * t.part_stride] = 0.f;
                }
            }
        }
    } else if (warp == kLoadWarp) {
        // ---- weights ----
        if (lane == 0) {
            st.par = 1;
            uint32_t n = 0;
            while (!dead && walk_next(a, wk, pc)) {
                const CUtensorMap *map = &a.map[pc.ten];
                for (uint32_t blk = pc.b0; blk < pc.b1; ++blk, ++n) {
                    if (!one_wait(smem + kEmpty + 8 * st.slot, st.par, a.status, abort_flag)) { dead = true; break; }
                    fence_proxy_async_smem();
                    uint64_t *full = bar_at(smem + kRawFull + 8 * st.slot);
                    mbar_arrive_expect_tx(full, kRows * kPitch);
                    // rows past the end of the tensor arrive as zeros
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                            stages + st.slot * kSlot<T>),
                        "l"(map), "r"(blk * 18u), "r"(pc.tile * kRows), "r"(smem_u32(full))
                        : "memory");
                    step_on();
                }
            }
            drain(kRawFull, n);
        }
    } else if (warp == kTensorWarp) {
        uint32_t buf = 0, apar = 0;
        Ring d[2] = {{0, 1}, {R / 2, 1}};   // the buffers of the epilogue's halves
        auto wait = [&](uint32_t bar, uint32_t parity) { return warp_wait(bar, parity, a.status, abort_flag); };
        while (!dead && walk_next(a, wk, pc)) {
            for (uint32_t blk = pc.b0; blk < pc.b1; ++blk) {
                Ring &r = d[buf];
                if (!wait(smem + kDEmpty + 8 * r.slot, r.par) || !wait(smem + kActFull + 8 * st.slot, st.par) || !wait(smem + kAFull + 8 * buf, apar)) { dead = true; break; }
                fence_after();
                const uint64_t b = b_desc(__shfl_sync(0xffffffffu, stages + st.slot * kSlot<T> + kRows * kPitch, 0));   // (uniform)
                const uint32_t at = __shfl_sync(0xffffffffu, tmem + kACol + buf * kABuf, 0), dt = __shfl_sync(0xffffffffu, tmem + kDCol + r.slot * (256 / R), 0);
                if (elect_one()) {
                    tensor_step<2 * T>(at, b, dt);
                    tm_commit(smem + kDFull + 8 * r.slot);
                    tm_commit(smem + kAEmpty + 8 * buf);
                }
                __syncwarp();
                if (R == 2) r.par ^= 1u;
                else if ((++r.slot & 1u) == 0) { r.slot -= 2; r.par ^= 1u; }
                buf ^= 1u;
                if (!buf) apar ^= 1u;
                step_on();
            }
        }
        if (dead) {   // nothing in flight when the tensor memory goes back
            if (elect_one()) tm_commit(smem + kDrain);
            __syncwarp();
            const uint64_t t0 = globaltimer_ns();
            while (!bar_try(smem + kDrain, 0) && globaltimer_ns() - t0 < kDefaultWaitNs) {}
        }
    } else if (warp == kTensorWarp + 1 && lane == 0) {
        // ---- the activation's image, step by step ----
        griddep_wait();
        st.par = 1;
        uint32_t n = 0;
        while (!dead && walk_next(a, wk, pc)) {
            for (uint32_t blk = pc.b0; blk < pc.b1; ++blk, ++n) {
                if (!one_wait(smem + kEmpty + 8 * st.slot, st.par, a.status, abort_flag)) { dead = true; break; }
                fence_proxy_async_smem();
                mbar_arrive_expect_tx(bar_at(smem + kActFull + 8 * st.slot), T * 1064u);
                bulk_g2s_addr(stages + st.slot * kSlot<T> + kRows * kPitch, a.xq + (size_t)blk * (T * 1064u), T * 1064u, bar_at(smem + kActFull + 8 * st.slot));
                step_on();
            }
        }
        drain(kActFull, n);
    }
    // every thread comes here, whatever happened; then the tensor memory goes back
    fence_before();
    __syncthreads();
    if (warp == kTensorWarp) {
        fence_after();
        asm volatile("tcgen05.dealloc.cta_group::1.sync.aligned.b32 %0, %1;" ::"r"(tmem), "r"(kTmemCols) : "memory");
    }
}

constexpr uint32_t kMaxParts = 8, kTmCtas = 148;

// The grid and the number of planes. A share of the line holds at least one step; with planes, no more than kMaxParts shares touch
// a tile: a tile's nblk steps start within nblk - 1 of each other, so that at most (nblk - 1) / share + 2 shares do.
struct TmPlan { uint32_t grid, parts, steps; };
bool tm_plan(const NxTensor *t, int n, uint32_t cols, bool split, TmPlan &p) {
    const uint32_t nblk = cols / 256;
    uint64_t tiles = 0;
    for (int i = 0; i < n; ++i) {
        if (t[i].fmt != FMT_Q4_K || t[i].rows == 0) return false;
        tiles += (t[i].rows + kRows - 1) / kRows;
    }
    if (tiles * nblk >= (1ull << 24)) return false;   // (shares are formed in 32 bits)
    p.steps = (uint32_t)tiles * nblk;
    if (!split) {
        p.grid = (uint32_t)std::min<uint64_t>(kTmCtas, tiles);
        p.parts = 1;
        return true;
    }
    p.grid = std::min(kTmCtas, p.steps);
    if (nblk > 1) p.grid = std::max(1u, std::min(p.grid, p.steps * (kMaxParts - 2) / (nblk - 1)));
    p.parts = p.grid == 1 ? 1 : std::min(kMaxParts, (nblk - 1) / (p.steps / p.grid) + 2);
    return true;
}

} // namespace

// FLB_UMMA=1 (read at every call, so that one process can run both kernels): every Q4_K call of several columns takes this form.
bool matmul_umma_on(void) {
    const char *v = getenv("FLB_UMMA");
    return v && v[0] == '1';
}

// Whether a launch whose planes are added on the fly takes this form. Time = start + steps per CTA x time of one, conversion included:
// 8 tokens 8.9 + 0.70 us against 7.9 + 0.84 (matvec_tc_nx.cu), 16 tokens 11.4 + 0.97 against 9.2 + 1.29, equal at 7 steps per CTA.
// Up to 4 tokens the other kernel needs half its tensor instructions and is the faster one (28672 x 4096, 2 tokens: 23.4
// against 23.9 us). Calls whose planes would take a launch of their own to add don't take it (14336 x 4096, 8 tokens: 17.4
// against 18.0 us, and 3 us for the planes).
bool matmul_tm_takes(const NxTensor *t, int n, uint32_t cols, uint32_t P) {
    TmPlan p;
    return P > 4 && tm_plan(t, n, cols, true, p) && p.grid == kTmCtas && p.steps >= 8 * kTmCtas;
}

uint32_t matmul_tm_parts(const NxTensor *t, int n, uint32_t cols, bool split) {
    TmPlan p;
    return tm_plan(t, n, cols, split, p) ? p.parts : 0;
}

cudaError_t matmul_tm_init(void) {
    const cudaError_t e = cudaFuncSetAttribute(matmul_tm_kernel<8>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
    return e != cudaSuccess ? e : cudaFuncSetAttribute(matmul_tm_kernel<16>, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
}

cudaError_t launch_tm_matmul(const NxIn &in, const NxTensor *t, int n, uint32_t cols, uint32_t P, int accumulate, const uint8_t *xq,
                             uint32_t *status, cudaStream_t stream, bool pdl, bool split) {
    TmPlan p;
    if (in.table || P == 0 || P > kNxMaxTokens || !tm_plan(t, n, cols, split, p) || (accumulate && p.parts > 1)) return cudaErrorNotSupported;
    TmArgs k;
    memset(&k, 0, sizeof(k));
    uint32_t base = 0;
    for (int i = 0; i < n; ++i) {
        TmT &d = k.t[i];
        d.y = t[i].y; d.part_stride = t[i].part_stride; d.rows = t[i].rows; d.ystride = t[i].ystride;
        d.base = base;
        const uint32_t pitch = t[i].pitch ? t[i].pitch : (uint32_t)row_bytes(FMT_Q4_K, cols);
        const cudaError_t e = tensor_map_2d(&k.map[i], 8, t[i].w, pitch / 8, t[i].rows, pitch, kPitch / 8, kRows, false);
        if (e != cudaSuccess) return e;
        base += (t[i].rows + kRows - 1) / kRows * (cols / 256);
    }
    k.n = n; k.steps = p.steps; k.nblk = cols / 256; k.P = P; k.parts = p.parts; k.whole = split ? 0 : 1;
    k.xq = xq; k.accumulate = accumulate; k.rms = in.wnorm ? 1 : 0; k.eps = in.eps; k.status = status;
    if (P > 8) return launch_kernel(matmul_tm_kernel<16>, dim3(p.grid), dim3(kThreads), head_of(16) + kSlots<16> * kSlot<16>, stream, pdl, k);
    return launch_kernel(matmul_tm_kernel<8>, dim3(p.grid), dim3(kThreads), head_of(8) + kSlots<8> * kSlot<8>, stream, pdl, k);
}

} // namespace flb
