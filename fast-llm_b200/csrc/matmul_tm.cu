// Several activation columns in one pass over Q4_K or Q6_K tensors on the Blackwell tensor cores: tcgen05.mma with the unpacked
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
//   unpack (2 x 4 warps)   : every other step each: packed bytes -> f16, written to tensor memory (Q4_K: thread = row)
//   epilogue (2 x 4 warps) : every other step (Q6_K: every other four results) each; thread = row: D out of tensor memory, scales
//                            and mins, sum over the steps in f32; the second hands its sums to the first at the end of a tile, which writes the results
//   weights (1 thread)     : the packed bytes of a step, one TMA box of 128 rows, into a ring of stages
//   activation (1 thread)  : the step's B operand (one bulk copy of the image that act_convert_nx_kernel built), same ring
//   tensor (1 warp)        : 16 instructions (M 128, N 2 x 8 or 2 x 16 tokens as (hi, lo), K 16) per step
// Every wait is bounded; a wait that runs out sets the status word and an abort flag all roles watch, the launch then drains,
// frees its tensor memory and returns.
//
// Arithmetic as in matvec_tc_nx.cu. Q6_K: q - 32 as f16, an instruction per scale group, scaled in f32 by the epilogue. Q4_K:
// (q - 8) sc as exact f16, activation of 22 bits per 256-column block, chains of four
// instructions (64 columns) from zero, added with rounding: tcgen05.mma truncates its running sum exactly as mma.sync does (bias of
// a chain of 4: -5.4e-8 of the result with either, of 16: -2.1e-7). The mins: 8 d sc - dmin m of a sub-block, rounded once, times
// the sub-block's f32 sum.
//
// What bounds it (B200): issue slots. A step of Q4_K with 8 tokens takes 2600 warp instructions besides the polls (324 per 16 rows;
// matvec_tc_nx.cu 413, 560 for 16 tokens), over four schedulers at 0.6 a cycle in the steady state; the tensor pipe is 8 % busy with 8
// tokens and 13 % with 16 (28672 x 4096 Q4_K; Q6_K 4 and 8 %; an instruction takes 15 cycles for N 16, 20 for N 32, with A in tensor
// memory; 40 with A in shared memory), the weights arrive at 5.9 TB/s when nothing else is done.
// 28672 x 4096 Q4_K with its conversion: 25.8 us for 8 tokens and 34.9 for 16 (matvec_tc_nx.cu: 28.3 and 40.5); 2 tokens 23.9 (23.4).
// Inside a pass more, since the activation arrives beside the weights instead of in front of them (70 KB per CTA): 8B shape, 16 tokens
// 4207 us with matvec_tc_nx.cu throughout, 3886 with gate | up, 3844 with O and 3626 with down (Q6_K) in this form too.
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
// Bytes of a row that a stage holds: odd multiples of 16, so that neither the row-per-thread reads nor the fragment reads of Q6_K
// collide. A Q6_K super-block (210 bytes) starts on any even byte; its stage starts on the 16-byte boundary in front of it.
__host__ __device__ constexpr uint32_t pitch_of(int fmt) { return fmt == FMT_Q4_K ? 144u : 240u; }

// A stage: the rows' bytes, then the step's activation (the operand's four tiles, sub-block sums, block scales, sums of squares).
template <int F, int T> constexpr uint32_t kSlot = (kRows * pitch_of(F) + T * 1064 + 1023) & ~1023u;
template <int F, int T> constexpr uint32_t kSlots = (kSmemLimit - head_of(T)) / kSlot<F, T> < kMaxSlots ? (kSmemLimit - head_of(T)) / kSlot<F, T> : kMaxSlots;
// The unpack groups take the steps in turn. A group that waits for step j has seen the tensor core take step j - 4, hence that and all before it
// landed: with four slots or more the slot's last stage is one of those, and the parity of its barrier tells the two apart.
static_assert(kSlots<FMT_Q4_K, 8> >= 4 && kSlots<FMT_Q4_K, 16> >= 4 && kSlots<FMT_Q6_K, 8> >= 4 && kSlots<FMT_Q6_K, 16> >= 4, "slots");

struct TmT {
    float *y;
    size_t part_stride;
    uint32_t rows, ystride, base;   // base: where the tensor starts on the line
};
struct TmArgs {
    CUtensorMap map[3];   // [rows][pitch / 8] 8-byte elements, box 128 rows x pitch_of
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
// 16 lanes x 64 columns of tensor memory from the warp: r[2 i], r[2 i + 1] = rows g, g + 8 of column 4 i + t
__device__ __forceinline__ void tm_store64(uint32_t addr, const uint32_t (&r)[32]) {
    asm volatile(
        "tcgen05.st.sync.aligned.16x128b.x16.b32 [%0], {%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15,%16,%17,%18,%19,%20,%21,%22,%23,"
        "%24,%25,%26,%27,%28,%29,%30,%31,%32};" ::"r"(addr),
        "r"(r[0]), "r"(r[1]), "r"(r[2]), "r"(r[3]), "r"(r[4]), "r"(r[5]), "r"(r[6]), "r"(r[7]), "r"(r[8]), "r"(r[9]), "r"(r[10]), "r"(r[11]),
        "r"(r[12]), "r"(r[13]), "r"(r[14]), "r"(r[15]), "r"(r[16]), "r"(r[17]), "r"(r[18]), "r"(r[19]), "r"(r[20]), "r"(r[21]), "r"(r[22]),
        "r"(r[23]), "r"(r[24]), "r"(r[25]), "r"(r[26]), "r"(r[27]), "r"(r[28]), "r"(r[29]), "r"(r[30]), "r"(r[31])
        : "memory");
}
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
// instructions: measured, one by one from a thread in a branch of its own an instruction cost 45 cycles alone and 135 beside the other
// roles, this way 15 (N 16).
__device__ __forceinline__ bool elect_one() {
    uint32_t r;
    asm volatile("{\n\t.reg .pred p;\n\telect.sync _|p, 0xffffffff;\n\tselp.u32 %0, 1, 0, p;\n\t}" : "=r"(r));
    return r != 0;
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }
__device__ __forceinline__ uint32_t hsub2_u32(uint32_t h, __half2 off) { return as_u32(__hsub2(as_h2(h), off)); }
__device__ __forceinline__ uint32_t hfma2_u32(uint32_t h, __half2 m, __half2 c) { return as_u32(__hfma2(as_h2(h), m, c)); }
// byte k of w as a float
__device__ __forceinline__ float u8f(uint32_t w, int k) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + k)) - 8388608.f; }
// byte k of w, which holds s + 128, as s
__device__ __forceinline__ float s8f(uint32_t w, int k) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + k)) - 8388736.f; }

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

// Steps of this CTA.
__device__ __forceinline__ uint32_t steps_of(const TmArgs &a) {
    const Walk w = walk_begin(a);
    return a.whole ? ((w.hi + a.nblk - 1) / a.nblk - (w.pos + a.nblk - 1) / a.nblk) * a.nblk : w.hi - w.pos;
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
// Q6_K, 16 rows at a time in the layout of an mma.sync A fragment, lane (g, t): rows g, g + 8 (r0: row g), column t of every four (a
// thread per row would have to realign its bytes by any even number). q - 32 as f16; instruction m = (2 hf + hq) * 4 + gq covers one
// scale group (matvec_tc_nx.cu). ODD: the block starts 2 bytes past a word boundary (r0 is 2 bytes in front of it).
template <bool ODD>
__device__ __forceinline__ void unpack_q6k(uint32_t r0, uint32_t t, uint32_t tm) {
    constexpr uint32_t kPitch = pitch_of(FMT_Q6_K);
    const __half2 off = __floats2half2_rn(1056.f, 1056.f);
#pragma unroll 1
    for (uint32_t hf = 0; hf < 2; ++hf) {
        uint32_t o[32];
#pragma unroll
        for (int hq = 0; hq < 2; ++hq)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t rb = r0 + r * 8 * kPitch, oa = 64 * hf + 16 * hq + 4 * t, oh = 128 + 32 * hf + 16 * hq + 4 * t;
                uint32_t a, b, h;
                if (ODD) {
                    a = __byte_perm(lds32(rb + oa), lds32(rb + oa + 4), 0x5432u);
                    b = __byte_perm(lds32(rb + oa + 32), lds32(rb + oa + 36), 0x5432u);
                    h = __byte_perm(lds32(rb + oh), lds32(rb + oh + 4), 0x5432u);
                } else {
                    a = lds32(rb + oa); b = lds32(rb + oa + 32); h = lds32(rb + oh);
                }
                uint32_t q[4];
                q[0] = (a & 0x0F0F0F0Fu) | ((h << 4) & 0x30303030u);
                q[1] = (b & 0x0F0F0F0Fu) | ((h << 2) & 0x30303030u);
                q[2] = ((a >> 4) & 0x0F0F0F0Fu) | (h & 0x30303030u);
                q[3] = ((b >> 4) & 0x0F0F0F0Fu) | ((h >> 2) & 0x30303030u);
#pragma unroll
                for (int gq = 0; gq < 4; ++gq) {   // bytes 0, 2 / 1, 3 under 0x64: f16 1024 + q
                    o[16 * hq + 4 * gq + r] = hsub2_u32(__byte_perm(q[gq], 0x64646464u, 0x4240u), off);
                    o[16 * hq + 4 * gq + 2 + r] = hsub2_u32(__byte_perm(q[gq], 0x64646464u, 0x4341u), off);
                }
            }
        tm_store64(tm + 64 * hf, o);
    }
}

// ---- epilogue of one step: acc[i] += the step's results of tokens 2 i, 2 i + 1 -----------------------------------------
// Four results at a time (D: 4 x N columns; N = 2 NT: hi columns of the tokens, then lo columns): Q4_K has one such unit per step, a
// half of the epilogue every other step; Q6_K four, a half every other one.
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
__device__ __forceinline__ bool epi_step_q4k(const Epi &e, Ring &d, uint32_t lane, uint32_t row_addr, uint32_t side, F2 (&acc)[NT / 2]) {
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

// Row address of the block's stage, which it starts `misalign` bytes into.
template <int NT, int R>
__device__ __forceinline__ bool epi_step_q6k(const Epi &e, Ring &d, uint32_t half, uint32_t lane, uint32_t row_addr, uint32_t misalign, uint32_t side, F2 (&acc)[NT / 2]) {
    // the 16 scales and d: 18 bytes from byte 192 of the block on
    const uint4 p0 = lds128(row_addr + 192), p1 = lds128(row_addr + 208);
    uint32_t w[8] = {p0.x, p0.y, p0.z, p0.w, p1.x, p1.y, p1.z, p1.w};
    if (misalign & 8u) {
#pragma unroll
        for (int k = 0; k < 6; ++k) w[k] = w[k + 2];
    }
    if (misalign & 4u) {
#pragma unroll
        for (int k = 0; k < 6; ++k) w[k] = w[k + 1];
    }
    if (misalign & 2u) {
#pragma unroll
        for (int k = 0; k < 5; ++k) w[k] = __byte_perm(w[k], w[k + 1], 0x5432u);
    }
    const F2 d2 = f2(h2f_bits((uint16_t)(w[4] & 0xFFFFu)));
#pragma unroll
    for (int k = 0; k < 4; ++k) w[k] ^= 0x80808080u;
    F2 sum[NT / 2];
#pragma unroll
    for (int i = 0; i < NT / 2; ++i) sum[i] = f2(0.f);
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {   // units 2 hf + half: the scale of group gq is 8 hf + 2 gq + half
        // The two parts of a group first, rounded at the group's size, then one rounding at that of the running sum: added one
        // after the other the error of 4096 x 14336 was 1.28e-7 (2-norm; matvec_tc_nx.cu 1.21e-7).
        const uint32_t lo = w[2 * hf] >> (8 * half), up = w[2 * hf + 1] >> (8 * half);
        const F2 f[4] = {f2(s8f(lo, 0)), f2(s8f(lo, 2)), f2(s8f(up, 0)), f2(s8f(up, 2))};
        const auto mul8 = [&](float (&a)[16], float (&b)[16], float (&c)[16], float (&g)[16]) {
#pragma unroll
            for (int i = 0; i < 4; ++i) {
                sum[i] = fma2(f[0], f2(a[2 * i], a[2 * i + 1]) + f2(a[8 + 2 * i], a[9 + 2 * i]), sum[i]);
                sum[i] = fma2(f[1], f2(b[2 * i], b[2 * i + 1]) + f2(b[8 + 2 * i], b[9 + 2 * i]), sum[i]);
                sum[i] = fma2(f[2], f2(c[2 * i], c[2 * i + 1]) + f2(c[8 + 2 * i], c[9 + 2 * i]), sum[i]);
                sum[i] = fma2(f[3], f2(g[2 * i], g[2 * i + 1]) + f2(g[8 + 2 * i], g[9 + 2 * i]), sum[i]);
            }
        };
        const auto mul16 = [&](int k, float (&h)[16], float (&l)[16]) {
#pragma unroll
            for (int i = 0; i < NT / 2; ++i) sum[i] = fma2(f[k], f2(h[2 * i], h[2 * i + 1]) + f2(l[2 * i], l[2 * i + 1]), sum[i]);
        };
        if constexpr (NT == 8) { if (!step_results<NT, R>(e, d, lane, mul8)) return false; }
        else { if (!step_results<NT, R>(e, d, lane, mul16)) return false; }
    }
#pragma unroll
    for (int i = 0; i < NT / 2; i += 2) {
        F2 x0, x1;
        lds_f2x2(side + NT * 32 + i * 8, x0, x1);
        // (never x0 d2 by itself: with an activation at either end of the range it is infinite or loses bits)
        acc[i] = fma2(x0, d2 * sum[i], acc[i]);
        acc[i + 1] = fma2(x1, d2 * sum[i + 1], acc[i + 1]);
    }
    return true;
}

// Instructions u .. of a step (a: its weights, b: descriptor of its activation) into a unit's four results at dt: all 16 of Q4_K, a chain
// of four each, or 4 of Q6_K's.
template <int F, int N>
__device__ __forceinline__ void tensor_unit(uint32_t a, uint64_t b, uint32_t dt, int u) {
    constexpr uint32_t idesc = (1u << 4) | ((N >> 3) << 17) | ((128u >> 4) << 24);   // f16 x f16 -> f32, K-major, M 128
    constexpr int C = F == FMT_Q4_K ? 4 : 1;
#pragma unroll
    for (int i = 0; i < 4 * C; ++i) {
        const int m = u + i;
        tm_mma(dt + i / C * N, a + 8 * m, b + (uint64_t)((m >> 2) * N * 8 + (m & 3) * 2), idesc, i % C);
    }
}

template <int F, int T>
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
            mbar_init(bar_at(smem + kEmpty + 8 * i), F == FMT_Q4_K ? 4 + 4 : 4 + 8);   // the step's unpack warps and epilogue (which comes after the tensor core)
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
    const uint32_t n_steps = steps_of(a);
    Piece pc;
    Ring st{0, 0};   // the stage ring
    auto step_on = [&]() { if (++st.slot == kSlots<F, T>) { st.slot = 0; st.par ^= 1u; } };
    bool dead = false;
    // after an abort: waits for the copies in flight, those of the last n steps of the ring's barriers at `full`
    auto drain = [&](uint32_t full, uint32_t n) {
        for (uint32_t k = 0; dead && k < min(n, kSlots<F, T>); ++k) {
            const uint32_t i = n - 1 - k;
            const uint64_t t0 = globaltimer_ns();
            while (!bar_try(smem + full + 8 * (i % kSlots<F, T>), (i / kSlots<F, T>) & 1u) && globaltimer_ns() - t0 < kDefaultWaitNs) {}
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
                const uint32_t raw = stages + st.slot * kSlot<F, T>;
                if (!warp_wait(smem + kRawFull + 8 * st.slot, st.par, a.status, abort_flag) ||
                    !warp_wait(smem + kAEmpty + 8 * wg, par, a.status, abort_flag)) { dead = true; break; }
                fence_after();
                const uint32_t tm = tmem + ((quad * 32) << 16) + kACol + wg * kABuf;
                if (F == FMT_Q4_K) unpack_q4k(raw + (quad * 32 + lane) * pitch_of(F), tm);
                else
#pragma unroll 1
                    for (uint32_t h = 0; h < 2; ++h) {
                        const uint32_t r0 = raw + (quad * 32 + 16 * h + (lane >> 2)) * pitch_of(F) + ((blk * 210u) & 15u);
                        if (blk & 1u) unpack_q6k<true>(r0 - 2, lane & 3u, tm + (h << 20));
                        else unpack_q6k<false>(r0, lane & 3u, tm + (h << 20));
                    }
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
                const uint32_t raw = stages + st.slot * kSlot<F, T>, side = raw + kRows * pitch_of(F) + T * 1024u;
                if (F == FMT_Q4_K && turn++ % 2 != half) { step_on(); continue; }
                if (!warp_wait(smem + kRawFull + 8 * st.slot, st.par, a.status, abort_flag) ||
                    !warp_wait(smem + kActFull + 8 * st.slot, st.par, a.status, abort_flag) ||
                    !(F == FMT_Q4_K ? epi_step_q4k<T, R>(e, d, lane, raw + row * pitch_of(F), side, acc)
                                    : epi_step_q6k<T, R>(e, d, half, lane, raw + row * pitch_of(F), (blk * 210u) & 15u, side, acc))) { dead = true; break; }
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
                    mbar_arrive_expect_tx(full, kRows * pitch_of(F));
                    const uint32_t x = F == FMT_Q4_K ? blk * 18u : ((blk * 210u) & ~15u) / 8;
                    // rows past the end of the tensor arrive as zeros
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                            stages + st.slot * kSlot<F, T>),
                        "l"(map), "r"(x), "r"(pc.tile * kRows), "r"(smem_u32(full))
                        : "memory");
                    step_on();
                }
            }
            drain(kRawFull, n);
        }
    } else if (warp == kTensorWarp) {
        uint32_t buf = 0, apar = 0, left = n_steps;
        Ring d[2] = {{0, 1}, {R / 2, 1}};   // the buffers of the epilogue's halves
        auto wait = [&](uint32_t bar, uint32_t parity) { return warp_wait(bar, parity, a.status, abort_flag); };
        while (!dead && walk_next(a, wk, pc)) {
            for (uint32_t blk = pc.b0; blk < pc.b1; ++blk) {
                if (!wait(smem + kActFull + 8 * st.slot, st.par) || !wait(smem + kAFull + 8 * buf, apar)) { dead = true; break; }
                fence_after();
                const uint64_t b = b_desc(__shfl_sync(0xffffffffu, stages + st.slot * kSlot<F, T> + kRows * pitch_of(F), 0));   // (uniform)
                const uint32_t at = __shfl_sync(0xffffffffu, tmem + kACol + buf * kABuf, 0);
#pragma unroll
                for (int u = 0; u < 16; u += F == FMT_Q4_K ? 16 : 4) {
                    Ring &r = d[F == FMT_Q4_K ? buf : (u >> 2) & 1];
                    if (!wait(smem + kDEmpty + 8 * r.slot, r.par)) { dead = true; break; }
                    fence_after();
                    const uint32_t dt = __shfl_sync(0xffffffffu, tmem + kDCol + r.slot * (256 / R), 0);
                    if (elect_one()) {
                        tensor_unit<F, 2 * T>(at, b, dt, u);
                        tm_commit(smem + kDFull + 8 * r.slot);
                    }
                    __syncwarp();
                    if (R == 2) r.par ^= 1u;
                    else if ((++r.slot & 1u) == 0) { r.slot -= 2; r.par ^= 1u; }
                }
                if (dead) break;
                // (not after the last step of either buffer: an arrival that nothing waits for could still be in flight when the CTA gives
                // its shared memory up to the next one, which may be there already as a programmatic dependent)
                if (left-- > 2 && elect_one()) tm_commit(smem + kAEmpty + 8 * buf);
                __syncwarp();
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
                bulk_g2s_addr(stages + st.slot * kSlot<F, T> + kRows * pitch_of(F), a.xq + (size_t)blk * (T * 1064u), T * 1064u, bar_at(smem + kActFull + 8 * st.slot));
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

constexpr uint32_t kMaxParts = 8;
static_assert(kMaxParts <= kMaxPlanes, "planes");

// The grid (a CTA per SM) and the number of planes. A share of the line holds at least one step; with planes, no more than kMaxParts shares touch
// a tile: a tile's nblk steps start within nblk - 1 of each other, so that at most (nblk - 1) / share + 2 shares do.
struct TmPlan { uint32_t grid, parts, steps; };
bool tm_plan(const NxTensor *t, int n, uint32_t cols, bool split, int sms, TmPlan &p) {
    const uint32_t nblk = cols / 256;
    uint64_t tiles = 0;
    for (int i = 0; i < n; ++i) {
        if ((t[i].fmt != FMT_Q4_K && t[i].fmt != FMT_Q6_K) || t[i].fmt != t[0].fmt || t[i].rows == 0) return false;
        tiles += (t[i].rows + kRows - 1) / kRows;
    }
    if (tiles * nblk >= (1ull << 24)) return false;   // (shares are formed in 32 bits)
    p.steps = (uint32_t)tiles * nblk;
    if (!split) {
        p.grid = (uint32_t)std::min<uint64_t>(sms, tiles);
        p.parts = 1;
        return true;
    }
    p.grid = std::min((uint32_t)sms, p.steps);
    if (nblk > 1) p.grid = std::max(1u, std::min(p.grid, p.steps * (kMaxParts - 2) / (nblk - 1)));
    p.parts = p.grid == 1 ? 1 : std::min(kMaxParts, (nblk - 1) / (p.steps / p.grid) + 2);
    return true;
}

} // namespace

// Read at every call, so that one process can run both kernels.
int matmul_tm_switch(void) {
    const char *v = getenv("FLB_UMMA");
    return v && v[0] >= '0' && v[0] <= '2' ? v[0] - '0' : -1;
}

// Whether a launch whose planes are added on the fly takes this form. Time of Q4_K alone = start + steps per CTA x time of one,
// conversion included: 8 tokens 8.9 + 0.70 us against 7.9 + 0.84 (matvec_tc_nx.cu), 16 tokens 11.4 + 0.97 against 9.2 + 1.29, equal at
// 7 steps per CTA. Inside a pass the line lies lower from 9 tokens on, since the other kernel's instance for so many is the slower one;
// passes of 8 layers over 512 keys (embedding / FFN) with this form over without it, 9 / 12 / 16 tokens:
//   4096 / 4096  Q4_K_M  (O and down, Q6_K, 3.5 steps per CTA, gate | up 6.9)  0.980 / 0.998 / 0.964
//   2048 / 8192  Q4_K    (down 3.5, gate | up 6.9)                             0.976 / 0.988 / 0.967
//   2048 / 14336 Q4_K_M  (down, Q6_K, 6.0, gate | up 12)                       0.977 / 0.979 / 0.953
// 5 and 8 tokens, from 8 steps on: 4096 / 10240 Q4_K_M (down, Q6_K, 8.6) 0.929 / 0.935, 2048 / 9472 Q4_K (gate | up 8.0) 0.968 / 0.969.
// Up to 4 tokens the other kernel needs half its tensor instructions and is the faster one alone (28672 x 4096, 2 tokens: 23.4 against
// 23.9 us), but not inside a pass (8B shape over 4096 keys, 2 / 3 / 4 tokens: 2968 / 3015 / 3060 us with it, 2938 / 2979 / 3048 with this
// form; at 8.0 to 8.6 steps, 2048 columns, 0.983 to 1.004). Calls whose planes would take a launch of their own to add don't take it
// (14336 x 4096, 8 tokens: 17.4 against 18.0 us, and 3 us for the planes).
bool matmul_tm_takes(const NxTensor *t, int n, uint32_t cols, uint32_t P, int sms) {
    TmPlan p;
    return P > 1 && tm_plan(t, n, cols, true, sms, p) && p.grid == (uint32_t)sms && p.steps >= (P > 8 ? 3 : 8) * p.grid;
}

// Whether the head of a pass, whose planes would take a reduction of their own, takes this form, a CTA whole tiles: from 9 columns on,
// where the other kernel cuts its 4096 columns in two and leaves planes, and from four tiles a CTA on, so that the last round of them is a small
// part. A pass of 16 positions: 6 layers, 90000 x 2560 Q4_K 657 -> 611 us, 12 positions 622 -> 590, 9 608 -> 581; 100000 x 1536 487 -> 463;
// 8B shape (128256 x 4096 Q6_K) 3605 -> 3565 (two boxes, with both forms in turn). Up to 8 columns the other kernel walks Q6_K in 131 us, this
// one's steps would take 165.
bool matmul_tm_takes_whole(const NxTensor *t, int n, uint32_t cols, uint32_t P, int sms) {
    TmPlan p;
    return P > 8 && tm_plan(t, n, cols, false, sms, p) && p.steps >= 4ull * (cols / 256) * sms;
}

uint32_t matmul_tm_parts(const NxTensor *t, int n, uint32_t cols, bool split, int sms) {
    TmPlan p;
    return tm_plan(t, n, cols, split, sms, p) ? p.parts : 0;
}

static const struct { void (*k)(const TmArgs); uint32_t smem; } kTmKernels[2][2] = {
    {{matmul_tm_kernel<FMT_Q4_K, 8>, head_of(8) + kSlots<FMT_Q4_K, 8> * kSlot<FMT_Q4_K, 8>}, {matmul_tm_kernel<FMT_Q4_K, 16>, head_of(16) + kSlots<FMT_Q4_K, 16> * kSlot<FMT_Q4_K, 16>}},
    {{matmul_tm_kernel<FMT_Q6_K, 8>, head_of(8) + kSlots<FMT_Q6_K, 8> * kSlot<FMT_Q6_K, 8>}, {matmul_tm_kernel<FMT_Q6_K, 16>, head_of(16) + kSlots<FMT_Q6_K, 16> * kSlot<FMT_Q6_K, 16>}}};

cudaError_t matmul_tm_init(void) {
    for (const auto &row : kTmKernels)
        for (const auto &k : row)
            if (const cudaError_t e = cudaFuncSetAttribute(k.k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)k.smem)) return e;
    return cudaSuccess;
}

cudaError_t launch_tm_matmul(const NxIn &in, const NxTensor *t, int n, uint32_t cols, uint32_t P, int accumulate, const uint8_t *xq,
                             uint32_t *status, int sms, cudaStream_t stream, bool pdl, bool split) {
    TmPlan p;
    if (in.table || P == 0 || P > kNxMaxTokens || !tm_plan(t, n, cols, split, sms, p) || (accumulate && p.parts > 1)) return cudaErrorNotSupported;
    TmArgs k;
    memset(&k, 0, sizeof(k));
    uint32_t base = 0;
    for (int i = 0; i < n; ++i) {
        TmT &d = k.t[i];
        d.y = t[i].y; d.part_stride = t[i].part_stride; d.rows = t[i].rows; d.ystride = t[i].ystride;
        d.base = base;
        const uint32_t pitch = t[i].pitch ? t[i].pitch : (uint32_t)row_bytes(t[i].fmt, cols);
        const cudaError_t e = tensor_map_2d(&k.map[i], 8, t[i].w, pitch / 8, t[i].rows, pitch, pitch_of(t[i].fmt) / 8, kRows, false);
        if (e != cudaSuccess) return e;
        base += (t[i].rows + kRows - 1) / kRows * (cols / 256);
    }
    k.n = n; k.steps = p.steps; k.nblk = cols / 256; k.P = P; k.parts = p.parts; k.whole = split ? 0 : 1;
    k.xq = xq; k.accumulate = accumulate; k.rms = in.wnorm ? 1 : 0; k.eps = in.eps; k.status = status;
    const auto &kernel = kTmKernels[t[0].fmt == FMT_Q6_K][P > 8];
    return launch_kernel(kernel.k, dim3(p.grid), dim3(kThreads), kernel.smem, stream, pdl, k);
}

} // namespace flb
