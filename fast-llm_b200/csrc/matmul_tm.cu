// Several activation columns in one pass over k-quant tensors on the Blackwell tensor cores: tcgen05.mma with the unpacked
// weights (A) and the results (D) in tensor memory, the activation (B) in shared memory. The same job as matvec_tc_nx.cu
// (Y[p][r] (+)= dot(W[r], X[p]), p < P <= 16; Q4_K, Q6_K, Q8_0; the STREAM_DOT semantics of Task::nx,
// include/fastllm/fastllm.h:87-96), whose tensor instructions bring every 16 x 16 weights into registers once per 4 tokens.
//
// Unit of work: a step = 128 rows x one 256-column super-block. The steps of all tensors (and experts) of a launch lie on
// one line, tile after tile, weighted by their bytes; every CTA takes an equal, contiguous piece of it. A tile that is
// shared by several CTAs leaves one plane of partial sums per CTA (planes that a tile does not need are written as zeros),
// which the next activation conversion adds in order: results are reproducible run to run.
//
// Roles of a CTA (16 warps), all coupled by mbarriers:
//   unpack (2 x 4 warps): every other step each: packed bytes -> f16, written to tensor memory in the layout of an mma.sync A
//                         fragment (tcgen05.st 16x128b: lane (g, t) holds rows g, g + 8, column t of every four)
//   epilogue (4 warps)  : thread = row: D out of tensor memory, scales, sum over the steps in f32, results
//   weights (1 thread)  : the packed bytes of a step, one TMA box of 128 rows, into a ring of stages
//   activation (1 thread): the step's B operand (one bulk copy of the image that act_convert_nx_kernel built), same ring
//   tensor (1 thread)   : 16 instructions (M 128, N 2 x tokens, K 16) per step
// Every wait is bounded; a wait that runs out sets the status word and an abort flag all roles watch, the launch then drains,
// frees its tensor memory and returns.
#include "common.cuh"
#include "kernels.h"

#include <algorithm>
#include <cstdlib>
#include <cstring>

namespace flb {

namespace {

constexpr uint32_t kRows = 128;
// 16 warps: four per quarter of the register file, 128 registers a thread
constexpr uint32_t kUnpackWarps = 8, kLoadWarp = 12, kTensorWarp = 13, kThreads = 16 * 32;   // the epilogue's from kUnpackWarps on
constexpr uint32_t kSmemLimit = 227 * 1024;
constexpr uint32_t kMaxSlots = 8, kHead = 1024;   // barriers in front of the ring
constexpr uint32_t kACol = 0, kABuf = 128, kDCol = 256, kTmemCols = 512;
// Bytes of a row that a stage holds: odd multiples of 16, so that neither the fragment reads of the unpack (8 rows x 4 lane
// columns) nor the row-per-thread reads of the epilogue collide. A Q6_K super-block (210 bytes) starts on any even byte; its
// stage starts on the 16-byte boundary in front of it.
__host__ __device__ constexpr uint32_t pitch_of(int fmt) { return fmt == FMT_Q4_K ? 144u : fmt == FMT_Q6_K ? 240u : 272u; }
__host__ __device__ constexpr uint32_t cost_of(int fmt) { return fmt == FMT_Q4_K ? 9u : fmt == FMT_Q6_K ? 13u : 17u; }   // a row's bytes of a step, roughly

struct TmT {
    float *y;
    size_t part_stride;
    uint32_t rows, ystride, tiles, xoff, base;   // base: where the tensor starts on the line of a group
    int fmt;
};
struct TmArgs {
    CUtensorMap map[3];   // [rows][pitch / 8] 8-byte elements, box 128 rows x pitch_of
    TmT t[3];
    uint32_t n, group_cost, group_grid, nblk, P, parts, whole;   // group_grid: the most CTAs that may share one group's line
    const uint8_t *xq;
    int accumulate, rms;
    float eps;
    uint32_t slots, slot_bytes, b_off;
    const uint32_t *table, *out_idx;
    uint32_t list_stride, col_off;
    int table_ready;
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
__device__ __forceinline__ uint32_t lds16(uint32_t addr) {
    uint16_t v;
    asm volatile("ld.shared.u16 %0, [%1];" : "=h"(v) : "r"(addr));
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
__device__ __noinline__ bool warp_wait_slow(uint32_t bar, uint32_t parity, uint32_t *status, volatile uint32_t *abort_flag) {
    const uint64_t t0 = globaltimer_ns();
    for (;;) {
        for (int i = 0; i < 64; ++i)
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
__device__ __noinline__ bool one_wait_slow(uint32_t bar, uint32_t parity, uint32_t *status, volatile uint32_t *abort_flag) {
    const uint64_t t0 = globaltimer_ns();
    for (;;) {
        for (int i = 0; i < 64; ++i)
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
__device__ __forceinline__ void tm_wait_st() { asm volatile("tcgen05.wait::st.sync.aligned;" ::: "memory"); }
// columns c .. c + 15 of this thread's lane; the values may be used after tm_wait_ld
__device__ __forceinline__ void tm_load16(uint32_t addr, float (&r)[16]) {
    asm volatile("tcgen05.ld.sync.aligned.32x32b.x16.b32 {%0,%1,%2,%3,%4,%5,%6,%7,%8,%9,%10,%11,%12,%13,%14,%15}, [%16];"
                 : "=f"(r[0]), "=f"(r[1]), "=f"(r[2]), "=f"(r[3]), "=f"(r[4]), "=f"(r[5]), "=f"(r[6]), "=f"(r[7]), "=f"(r[8]), "=f"(r[9]),
                   "=f"(r[10]), "=f"(r[11]), "=f"(r[12]), "=f"(r[13]), "=f"(r[14]), "=f"(r[15])
                 : "r"(addr)
                 : "memory");
}
// waits for the loads of four results; names them, so that nothing uses them earlier
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
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }
__device__ __forceinline__ uint32_t hsub2_u32(uint32_t h, __half2 off) { return as_u32(__hsub2(as_h2(h), off)); }
__device__ __forceinline__ uint32_t hfma2_u32(uint32_t h, __half2 m, __half2 c) { return as_u32(__hfma2(as_h2(h), m, c)); }
// byte k of w as a float; byte k of w, which holds s + 128, as s
__device__ __forceinline__ float u8f(uint32_t w, int k) { return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + k)) - 8388608.f; }
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
struct Piece { uint32_t ten, tile, b0, b1, n_valid, grp, row0, unit0, plane; };
struct Walk { uint32_t pos, hi, W, G; };   // G: CTAs that share the line
__device__ __forceinline__ uint32_t share_lo(const Walk &w, uint32_t c) { return w.W / w.G * c + w.W % w.G * c / w.G; }
__device__ __forceinline__ Walk walk_begin(const TmArgs &a) {
    Walk w;
    const uint32_t n_act = a.table ? a.table[0] : 1u;
    w.W = a.group_cost * n_act;
    w.G = max(1u, min(gridDim.x, a.group_grid * n_act));
    w.pos = share_lo(w, min(blockIdx.x, w.G));
    w.hi = share_lo(w, min(blockIdx.x + 1, w.G));
    return w;
}
__device__ __noinline__ bool walk_next(const TmArgs &a, Walk &w, Piece &p) {
    for (;;) {
        if (w.pos >= w.hi) return false;
        const uint32_t g = w.pos / a.group_cost, r = w.pos - g * a.group_cost;
        uint32_t j = 0;
        if (a.n > 1 && r >= a.t[1].base) j = 1;
        if (a.n > 2 && r >= a.t[2].base) j = 2;
        const TmT &t = a.t[j];
        const uint32_t c = cost_of(t.fmt), base = g * a.group_cost + t.base, total = t.tiles * a.nblk;
        uint32_t st = (r - t.base + c - 1) / c;   // the first step that starts here or later
        if (a.whole) st = (st + a.nblk - 1) / a.nblk * a.nblk;
        if (st >= total) { w.pos = base + total * c; continue; }
        const uint32_t start = base + st * c;
        if (start >= w.hi) return false;
        p.ten = j; p.tile = st / a.nblk; p.b0 = st - p.tile * a.nblk;
        p.b1 = a.whole ? a.nblk : min(a.nblk, p.b0 + (w.hi - start + c - 1) / c);
        w.pos = start + (p.b1 - p.b0) * c;
        p.plane = 0;
        if (p.b0) {   // the CTAs in front that have steps of this tile
            const uint32_t first = start - p.b0 * c;
            p.plane = 1;
            while (share_lo(w, blockIdx.x - p.plane) > first) ++p.plane;
        }
        p.n_valid = a.P; p.grp = 0; p.row0 = 0; p.unit0 = 0;
        if (a.table) {
            const uint4 e = reinterpret_cast<const uint4 *>(a.table)[1 + g];
            p.grp = e.x; p.n_valid = e.y; p.unit0 = e.z >> 16; p.row0 = e.w;
        }
        return true;
    }
}

// Offsets in shared memory.
constexpr uint32_t kRawFull = 0, kActFull = kRawFull + 8 * kMaxSlots, kEmpty = kActFull + 8 * kMaxSlots, kAFull = kEmpty + 8 * kMaxSlots,
                   kAEmpty = kAFull + 16, kDFull = kAEmpty + 16, kDEmpty = kDFull + 32, kDrain = kDEmpty + 32, kTmemPtr = kDrain + 8,
                   kAbort = kTmemPtr + 4;
static_assert(kAbort + 4 <= kHead, "head");

// ---- unpack: 16 rows x 256 columns of a warp (lane (g, t): rows g, g + 8) into 128 columns of tensor memory -----------
// Q4_K, r0: the row g of the 16. Arithmetic as in matvec_tc_nx.cu: a masked nibble is the subnormal f16 q 2^-24 (q 2^-20 in
// the high nibble), one FMA makes it (q - 8) sc 2^-14, exact. Lane column t takes the 32-byte chunk t; instruction m = 2 j + hb
// covers word j of every chunk, low (hb = 0) or high nibbles.
__device__ __forceinline__ void unpack_q4k(uint32_t r0, uint32_t t, uint32_t tm) {
    constexpr uint32_t kPitch = pitch_of(FMT_Q4_K);
    const uint32_t r1 = r0 + 8 * kPitch;
    uint4 hd[2], wd[2][2];
    hd[0] = lds128(r0); hd[1] = lds128(r1);
    wd[0][0] = lds128(r0 + 16 + 32 * t); wd[0][1] = lds128(r1 + 16 + 32 * t);
    wd[1][0] = lds128(r0 + 32 + 32 * t); wd[1][1] = lds128(r1 + 32 + 32 * t);
    // 6-bit scales of sub-blocks 2 t, 2 t + 1 (packing: fl_q4k_scale_min, src/runtime/quants.h:121-129)
    const uint32_t sh = 16u * (t & 1u);
    const uint32_t shA = t >= 2 ? sh + 2u : sh, mA = t >= 2 ? 0x3030u : 0x3F3Fu, mE = t >= 2 ? 0x0F0Fu : 0u;
    __half2 sL[2], sH[2], kL[2], kH[2];   // scales times 2^10 (low nibbles), 2^6 (high nibbles); -8 2^-14 times the scales
    const __half2 k1024 = __floats2half2_rn(1024.f, 1024.f), k64 = __floats2half2_rn(64.f, 64.f);
    const __half2 km8 = __floats2half2_rn(-0.00048828125f, -0.00048828125f);   // -8 2^-14
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t sc = ((hd[r].y >> shA) & mA) | ((hd[r].w >> sh) & mE);
        const __half2 s0 = __hsub2(as_h2(__byte_perm(sc, 0x64646464u, 0x4040u)), k1024), s1 = __hsub2(as_h2(__byte_perm(sc, 0x64646464u, 0x4141u)), k1024);
        sL[r] = __hmul2(s0, k1024); kL[r] = __hmul2(s0, km8);
        sH[r] = __hmul2(s1, k64); kH[r] = __hmul2(s1, km8);
    }
    const uint32_t ML = 0x000F000Fu, MH = 0x00F000F0u;
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        uint32_t o[32];
#pragma unroll
        for (int j = 0; j < 4; ++j)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint4 &q = wd[half][r];
                const uint32_t W = j == 0 ? q.x : j == 1 ? q.y : j == 2 ? q.z : q.w, V = W >> 8;
                o[8 * j + r] = hfma2_u32(W & ML, sL[r], kL[r]);
                o[8 * j + 2 + r] = hfma2_u32(V & ML, sL[r], kL[r]);
                o[8 * j + 4 + r] = hfma2_u32(W & MH, sH[r], kH[r]);
                o[8 * j + 6 + r] = hfma2_u32(V & MH, sH[r], kH[r]);
            }
        tm_store64(tm + 64 * half, o);
    }
}
// Q6_K: q - 32 as f16; instruction m = (2 hf + hq) * 4 + gq covers one scale group (matvec_tc_nx.cu). ODD: the block starts 2 bytes
// past a word boundary (r0 is 2 bytes in front of it).
template <bool ODD>
__device__ __forceinline__ void unpack_q6k(uint32_t r0, uint32_t t, uint32_t tm) {
    constexpr uint32_t kPitch = pitch_of(FMT_Q6_K);
    const __half2 off = __floats2half2_rn(1056.f, 1056.f);
#pragma unroll
    for (int hf = 0; hf < 2; ++hf) {
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
                for (int gq = 0; gq < 4; ++gq) {
                    o[16 * hq + 4 * gq + r] = hsub2_u32(__byte_perm(q[gq], 0x64646464u, 0x4240u), off);
                    o[16 * hq + 4 * gq + 2 + r] = hsub2_u32(__byte_perm(q[gq], 0x64646464u, 0x4341u), off);
                }
            }
        tm_store64(tm + 64 * hf, o);
    }
}
// Q8_0: instruction m = 2 b + i covers bytes 8 t + 4 i .. + 3 of block b for the lane columns t.
__device__ __forceinline__ void unpack_q80(uint32_t r0, uint32_t t, uint32_t tm) {
    constexpr uint32_t kPitch = pitch_of(FMT_Q8_0);
    const __half2 off = __floats2half2_rn(1152.f, 1152.f);
#pragma unroll
    for (int half = 0; half < 2; ++half) {
        uint32_t o[32];
#pragma unroll
        for (int bp = 0; bp < 2; ++bp)   // pairs of blocks: 68 bytes; even blocks' quants are 2 bytes past a word boundary
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                const uint32_t q = r0 + r * 8 * kPitch + 68 * (2 * half + bp) + 8 * t;
                const uint32_t x0 = lds32(q), x1 = lds32(q + 4), x2 = lds32(q + 8);
                uint32_t w[4];
                w[0] = __byte_perm(x0, x1, 0x5432u) ^ 0x80808080u;
                w[1] = __byte_perm(x1, x2, 0x5432u) ^ 0x80808080u;
                w[2] = lds32(q + 36) ^ 0x80808080u;
                w[3] = lds32(q + 40) ^ 0x80808080u;
#pragma unroll
                for (int i = 0; i < 4; ++i) {   // (block of the pair, half of the block)
                    o[16 * bp + 4 * i + r] = hsub2_u32(__byte_perm(w[i], 0x64646464u, 0x4240u), off);
                    o[16 * bp + 4 * i + 2 + r] = hsub2_u32(__byte_perm(w[i], 0x64646464u, 0x4341u), off);
                }
            }
        tm_store64(tm + 64 * half, o);
    }
}

// ---- epilogue of one step: acc[i] += the step's results of tokens 2 i, 2 i + 1 -----------------------------------------
// The four results of a unit (D: 4 x N columns at d; N = 2 NT: hi columns of the tokens, then lo columns). NT 8: a result is
// one load of 16, NT 16: two.
struct Ring { uint32_t slot, par; };
struct Epi {
    uint32_t smem, tmem;   // tmem: this warp's lanes
    uint32_t *status, *abort_flag;
};
template <int NT, int R, typename F>
__device__ __forceinline__ bool unit_results(const Epi &e, Ring &d, uint32_t lane, F &&use) {
    if (!warp_wait(e.smem + kDFull + 8 * d.slot, d.par, e.status, e.abort_flag)) return false;
    fence_after();
    const uint32_t at = e.tmem + kDCol + d.slot * (256 / R);
    float r0[16], r1[16], r2[16], r3[16];
    tm_load16(at, r0); tm_load16(at + 2 * NT, r1); tm_load16(at + 4 * NT, r2); tm_load16(at + 6 * NT, r3);
    tm_wait_ld(r0, r1, r2, r3);
    if (NT == 8) {
        fence_before();
        __syncwarp();
        if (lane == 0) bar_arrive(e.smem + kDEmpty + 8 * d.slot);
    }
    use(0, r0, r1, r2, r3);
    if (NT == 16) {
        tm_load16(at + 16, r0); tm_load16(at + 48, r1); tm_load16(at + 80, r2); tm_load16(at + 112, r3);
        tm_wait_ld(r0, r1, r2, r3);
        fence_before();
        __syncwarp();
        if (lane == 0) bar_arrive(e.smem + kDEmpty + 8 * d.slot);
        use(1, r0, r1, r2, r3);
    }
    if (++d.slot == R) { d.slot = 0; d.par ^= 1u; }
    return true;
}
template <int FMT, int NT, int R>
__device__ __forceinline__ bool epi_step(const Epi &e, Ring &d, uint32_t lane, uint32_t row_addr, uint32_t misalign, uint32_t side, F2 (&acc)[NT / 2]) {
    const uint32_t xs = side + NT * 32;
    F2 sum[NT / 2];
    if constexpr (FMT == FMT_Q4_K) {
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
        if (!unit_results<NT, R>(e, d, lane, [&](int part, float (&a)[16], float (&b)[16], float (&c)[16], float (&f)[16]) {
#pragma unroll
                for (int i = 0; i < NT / 2; ++i) {
                    F2 s = (f2(a[2 * i], a[2 * i + 1]) + f2(b[2 * i], b[2 * i + 1])) + (f2(c[2 * i], c[2 * i + 1]) + f2(f[2 * i], f[2 * i + 1]));
                    if constexpr (NT == 8) s = s + ((f2(a[8 + 2 * i], a[9 + 2 * i]) + f2(b[8 + 2 * i], b[9 + 2 * i])) + (f2(c[8 + 2 * i], c[9 + 2 * i]) + f2(f[8 + 2 * i], f[9 + 2 * i])));
                    sum[i] = part ? sum[i] + s : s;
                }
            })) return false;
#pragma unroll
        for (int i = 0; i < NT / 2; i += 2) {
            F2 x0, x1;
            lds_f2x2(xs + i * 8, x0, x1);
            acc[i] = fma2(x0, fma2(dq, sum[i], v[i]), acc[i]);
            acc[i + 1] = fma2(x1, fma2(dq, sum[i + 1], v[i + 1]), acc[i + 1]);
        }
    } else {
#pragma unroll
        for (int i = 0; i < NT / 2; ++i) sum[i] = f2(0.f);
        auto add4 = [&](float s0, float s1, float s2, float s3) {
            const F2 f0 = f2(s0), f1 = f2(s1), f2_ = f2(s2), f3 = f2(s3);
            return unit_results<NT, R>(e, d, lane, [&](int, float (&a)[16], float (&b)[16], float (&c)[16], float (&f)[16]) {
#pragma unroll
                for (int i = 0; i < NT / 2; ++i) {
                    sum[i] = fma2(f0, f2(a[2 * i], a[2 * i + 1]), sum[i]);
                    sum[i] = fma2(f1, f2(b[2 * i], b[2 * i + 1]), sum[i]);
                    sum[i] = fma2(f2_, f2(c[2 * i], c[2 * i + 1]), sum[i]);
                    sum[i] = fma2(f3, f2(f[2 * i], f[2 * i + 1]), sum[i]);
                    if constexpr (NT == 8) {
                        sum[i] = fma2(f0, f2(a[8 + 2 * i], a[9 + 2 * i]), sum[i]);
                        sum[i] = fma2(f1, f2(b[8 + 2 * i], b[9 + 2 * i]), sum[i]);
                        sum[i] = fma2(f2_, f2(c[8 + 2 * i], c[9 + 2 * i]), sum[i]);
                        sum[i] = fma2(f3, f2(f[8 + 2 * i], f[9 + 2 * i]), sum[i]);
                    }
                }
            });
        };
        float dd = 1.f;
        if constexpr (FMT == FMT_Q6_K) {
            // the 16 scales and d: 18 bytes from byte 192 of the block on, which lies `misalign` bytes into its stage
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
            dd = h2f_bits((uint16_t)(w[4] & 0xFFFFu));
#pragma unroll
            for (int k = 0; k < 4; ++k) w[k] ^= 0x80808080u;
#pragma unroll
            for (int hh = 0; hh < 4; ++hh) {
                const int s = 8 * (hh >> 1) + (hh & 1);   // scale of group gq: s + 2 gq
                if (!add4(s8f(w[s >> 2], s & 3), s8f(w[(s + 2) >> 2], (s + 2) & 3), s8f(w[(s + 4) >> 2], (s + 4) & 3), s8f(w[(s + 6) >> 2], (s + 6) & 3))) return false;
            }
        } else {
#pragma unroll
            for (int h = 0; h < 2; ++h) {
                float s[4];
#pragma unroll
                for (int k = 0; k < 4; ++k) s[k] = h2f_bits((uint16_t)lds16(row_addr + 34 * (4 * h + k)));
                if (!add4(s[0], s[1], s[2], s[3])) return false;
            }
        }
        const F2 d2 = f2(dd);
#pragma unroll
        for (int i = 0; i < NT / 2; i += 2) {
            F2 x0, x1;
            lds_f2x2(xs + i * 8, x0, x1);
            if (FMT == FMT_Q6_K) { x0 = x0 * d2; x1 = x1 * d2; }
            acc[i] = fma2(x0, sum[i], acc[i]);
            acc[i + 1] = fma2(x1, sum[i + 1], acc[i + 1]);
        }
    }
    return true;
}

// The 16 instructions of a step (a: its weights, b: descriptor of its activation): a result is the sum of 1 << CHAIN of them, a
// unit four results.
template <int CHAIN, int R, typename W>
__device__ __forceinline__ bool tensor_step(uint32_t a, uint64_t b, uint32_t d0, uint32_t N, uint32_t idesc, Ring &d, uint32_t smem, W &&wait) {
#pragma unroll
    for (int u = 0; u < 16; u += 4 << CHAIN) {
        if (!wait(smem + kDEmpty + 8 * d.slot, d.par)) return false;
        fence_after();
        const uint32_t dt = d0 + d.slot * (256 / R);
#pragma unroll
        for (int i = 0; i < 4 << CHAIN; ++i)
            tm_mma(dt + (i >> CHAIN) * N, a + 8 * (u + i), b + (uint64_t)(((u + i) >> 2) * N * 8 + ((u + i) & 3) * 2), idesc, i & ((1 << CHAIN) - 1));
        tm_commit(smem + kDFull + 8 * d.slot);
        if (++d.slot == R) { d.slot = 0; d.par ^= 1u; }
    }
    return true;
}

template <int FM, int T>
__global__ void __launch_bounds__(kThreads, 1) matmul_tm_kernel(const __grid_constant__ TmArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr int R = T == 16 ? 2 : 4;   // D buffers (4 x N columns each)
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5, smem = smem_u32(smem_raw);
    uint32_t *abort_flag = reinterpret_cast<uint32_t *>(smem_raw + kAbort);
    griddep_launch_dependents();
    if (a.table && !a.table_ready) griddep_wait();
    if (tid == 0) {
        for (uint32_t i = 0; i < kMaxSlots; ++i) {
            mbar_init(bar_at(smem + kRawFull + 8 * i), 1);
            mbar_init(bar_at(smem + kActFull + 8 * i), 1);
            mbar_init(bar_at(smem + kEmpty + 8 * i), 4 + 4 + 1);   // the unpack warps of the step, the epilogue, the tensor core
        }
        for (uint32_t i = 0; i < 2; ++i) { mbar_init(bar_at(smem + kAFull + 8 * i), 4); mbar_init(bar_at(smem + kAEmpty + 8 * i), 1); }
        for (uint32_t i = 0; i < (uint32_t)R; ++i) { mbar_init(bar_at(smem + kDFull + 8 * i), 1); mbar_init(bar_at(smem + kDEmpty + 8 * i), 4); }
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
    const uint32_t tmem = lds32(smem + kTmemPtr), stages = smem + kHead;
    Walk wk = walk_begin(a);
    Piece pc;
    Ring st{0, 0};   // the stage ring
    auto step_on = [&]() { if (++st.slot == a.slots) { st.slot = 0; st.par ^= 1u; } };
    bool dead = false;
    // after an abort: waits for the copies in flight, those of the last n steps of the ring's barriers at `full`
    auto drain = [&](uint32_t full, uint32_t n) {
        for (uint32_t k = 0; dead && k < min(n, a.slots); ++k) {
            const uint32_t i = n - 1 - k;
            const uint64_t t0 = globaltimer_ns();
            while (!bar_try(smem + full + 8 * (i % a.slots), (i / a.slots) & 1u) && globaltimer_ns() - t0 < kDefaultWaitNs) {}
        }
    };

    if (warp < kUnpackWarps) {
        const uint32_t wg = warp >> 2, quad = warp & 3u, g = lane >> 2, t = lane & 3u;
        uint32_t turn = 0, par = 1;   // a fresh barrier passes a wait on parity 1
        while (!dead && walk_next(a, wk, pc)) {
            const int fmt = a.t[pc.ten].fmt;
            for (uint32_t blk = pc.b0; blk < pc.b1; ++blk, turn ^= 1u) {
                if (turn != wg) { step_on(); continue; }
                const uint32_t raw = stages + st.slot * a.slot_bytes;
                if (!warp_wait(smem + kRawFull + 8 * st.slot, st.par, a.status, abort_flag) ||
                    !warp_wait(smem + kAEmpty + 8 * wg, par, a.status, abort_flag)) { dead = true; break; }
                fence_after();
#pragma unroll 1
                for (uint32_t h = 0; h < 2; ++h) {
                    const uint32_t row = quad * 32 + 16 * h + g, tm = tmem + ((quad * 32 + 16 * h) << 16) + kACol + wg * kABuf;
                    if ((FM & 1) && (FM == 1 || fmt == FMT_Q4_K)) unpack_q4k(raw + row * pitch_of(FMT_Q4_K), t, tm);
                    else if ((FM & 2) && (FM == 2 || fmt == FMT_Q6_K)) {
                        const uint32_t r0 = raw + row * pitch_of(FMT_Q6_K) + ((blk * 210u) & 15u);
                        if (blk & 1u) unpack_q6k<true>(r0 - 2, t, tm);
                        else unpack_q6k<false>(r0, t, tm);
                    } else if (FM & 4) unpack_q80(raw + row * pitch_of(FMT_Q8_0), t, tm);
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
        const Epi e{smem, tmem + ((quad * 32) << 16), a.status, abort_flag};
        Ring d{0, 0};
        griddep_wait();   // y and the sums of squares come from the kernels before
        float inv = 1.f;
        uint32_t inv_of = 0xFFFFFFFFu;
        while (!dead && walk_next(a, wk, pc)) {
            const TmT &t = a.t[pc.ten];
            const uint32_t nt = T == 16 && pc.n_valid > 8 ? 16u : 8u, xb = nt * 1064u;
            if (a.rms && inv_of != pc.grp) {   // lane p: 1 / rms of token p
                const uint8_t *ss_at = a.xq + t.xoff + (size_t)pc.unit0 * a.nblk * kTmUnit + nt * 1060u + (lane & (nt - 1)) * 4u;
                float ss = 0.f;
#pragma unroll 8
                for (uint32_t b = 0; b < a.nblk; ++b) ss += __ldcg(reinterpret_cast<const float *>(ss_at + (size_t)b * xb));
                inv = 1.0f / sqrtf(ss / (float)(a.nblk * 256u) + a.eps);
                inv_of = pc.grp;
            }
            F2 acc[T / 2];
#pragma unroll
            for (int i = 0; i < T / 2; ++i) acc[i] = f2(0.f);
            const int fmt = t.fmt;
            for (uint32_t blk = pc.b0; blk < pc.b1; ++blk) {
                const uint32_t raw = stages + st.slot * a.slot_bytes, side = raw + a.b_off + nt * 1024u;
                if (!warp_wait(smem + kRawFull + 8 * st.slot, st.par, a.status, abort_flag) ||
                    !warp_wait(smem + kActFull + 8 * st.slot, st.par, a.status, abort_flag)) { dead = true; break; }
                bool ok = true;
#define FLB_EPI(F, N) epi_step<F, N, R>(e, d, lane, raw + row * pitch_of(F), F == FMT_Q6_K ? (blk * 210u) & 15u : 0u, side, reinterpret_cast<F2(&)[N / 2]>(acc))
#define FLB_EPI_N(F) (T == 8 || nt == 8 ? FLB_EPI(F, 8) : FLB_EPI(F, T))
                if ((FM & 1) && (FM == 1 || fmt == FMT_Q4_K)) ok = FLB_EPI_N(FMT_Q4_K);
                else if ((FM & 2) && (FM == 2 || fmt == FMT_Q6_K)) ok = FLB_EPI_N(FMT_Q6_K);
                else if (FM & 4) ok = FLB_EPI_N(FMT_Q8_0);
#undef FLB_EPI_N
#undef FLB_EPI
                if (!ok) { dead = true; break; }
                __syncwarp();
                if (lane == 0) bar_arrive(smem + kEmpty + 8 * st.slot);
                step_on();
            }
            if (dead) break;
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
                    if (p >= pc.n_valid) continue;
                    const size_t orow = a.out_idx ? a.out_idx[(size_t)pc.grp * a.list_stride + a.col_off + p] : pc.row0 + p;
                    if (!in) continue;
                    float *dst = plane + orow * t.ystride;
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
                const TmT &t = a.t[pc.ten];
                const CUtensorMap *map = &a.map[pc.ten];
                const uint32_t row0 = pc.grp * t.rows + pc.tile * kRows, bytes = kRows * pitch_of(t.fmt);
                const int fmt = t.fmt;
                for (uint32_t blk = pc.b0; blk < pc.b1; ++blk, ++n) {
                    if (!one_wait(smem + kEmpty + 8 * st.slot, st.par, a.status, abort_flag)) { dead = true; break; }
                    fence_proxy_async_smem();
                    uint64_t *full = bar_at(smem + kRawFull + 8 * st.slot);
                    mbar_arrive_expect_tx(full, bytes);
                    // rows past the end of the tensor arrive as zeros (or as another expert's rows, whose results are dropped)
                    const uint32_t x = fmt == FMT_Q4_K ? blk * 18u : fmt == FMT_Q6_K ? ((blk * 210u) & ~15u) / 8 : blk * 34u;
                    asm volatile(
                        "cp.async.bulk.tensor.2d.shared::cluster.global.tile.mbarrier::complete_tx::bytes [%0], [%1, {%2, %3}], [%4];" ::"r"(
                            stages + st.slot * a.slot_bytes),
                        "l"(map), "r"(x), "r"(row0), "r"(smem_u32(full))
                        : "memory");
                    step_on();
                }
            }
            drain(kRawFull, n);
        }
    } else if (warp == kTensorWarp) {
        if (lane == 0) {
            uint32_t buf = 0, apar = 0;
            Ring d{0, 1};
            while (!dead && walk_next(a, wk, pc)) {
                const int fmt = a.t[pc.ten].fmt;
                const uint32_t nt = T == 16 && pc.n_valid > 8 ? 16u : 8u, N = 2 * nt;
                const uint32_t idesc = (1u << 4) | ((N >> 3) << 17) | ((128u >> 4) << 24);
                for (uint32_t blk = pc.b0; blk < pc.b1 && !dead; ++blk) {
                    if (!one_wait(smem + kActFull + 8 * st.slot, st.par, a.status, abort_flag) ||
                        !one_wait(smem + kAFull + 8 * buf, apar, a.status, abort_flag)) { dead = true; break; }
                    fence_after();
                    const uint64_t b = b_desc(stages + st.slot * a.slot_bytes + a.b_off);
                    const uint32_t at = tmem + kACol + buf * kABuf;
                    auto wait = [&](uint32_t bar, uint32_t parity) { return one_wait(bar, parity, a.status, abort_flag); };
                    if ((FM & 1) && (FM == 1 || fmt == FMT_Q4_K)) dead = !tensor_step<2, R>(at, b, tmem + kDCol, N, idesc, d, smem, wait);
                    else if ((FM & 2) && (FM == 2 || fmt == FMT_Q6_K)) dead = !tensor_step<0, R>(at, b, tmem + kDCol, N, idesc, d, smem, wait);
                    else if (FM & 4) dead = !tensor_step<1, R>(at, b, tmem + kDCol, N, idesc, d, smem, wait);
                    if (dead) break;
                    tm_commit(smem + kAEmpty + 8 * buf);
                    tm_commit(smem + kEmpty + 8 * st.slot);
                    buf ^= 1u;
                    if (!buf) apar ^= 1u;
                    step_on();
                }
            }
            if (dead) {   // nothing in flight when the tensor memory goes back
                tm_commit(smem + kDrain);
                const uint64_t t0 = globaltimer_ns();
                while (!bar_try(smem + kDrain, 0) && globaltimer_ns() - t0 < kDefaultWaitNs) {}
            }
        }
    } else if (warp == kTensorWarp + 1 && lane == 0) {
        // ---- the activation's image, step by step ----
        griddep_wait();
        st.par = 1;
        uint32_t n = 0;
        while (!dead && walk_next(a, wk, pc)) {
            const uint32_t nt = T == 16 && pc.n_valid > 8 ? 16u : 8u, xb = nt * 1064u;
            const uint8_t *img = a.xq + a.t[pc.ten].xoff + (size_t)pc.unit0 * a.nblk * kTmUnit;
            for (uint32_t blk = pc.b0; blk < pc.b1; ++blk, ++n) {
                if (!one_wait(smem + kEmpty + 8 * st.slot, st.par, a.status, abort_flag)) { dead = true; break; }
                fence_proxy_async_smem();
                mbar_arrive_expect_tx(bar_at(smem + kActFull + 8 * st.slot), xb);
                bulk_g2s_addr(stages + st.slot * a.slot_bytes + a.b_off, img + (size_t)blk * xb, xb, bar_at(smem + kActFull + 8 * st.slot));
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

void (*const kTmKernels[2][5])(const TmArgs) = {
    {matmul_tm_kernel<1, 8>, matmul_tm_kernel<2, 8>, matmul_tm_kernel<3, 8>, matmul_tm_kernel<4, 8>, matmul_tm_kernel<7, 8>},
    {matmul_tm_kernel<1, 16>, matmul_tm_kernel<2, 16>, matmul_tm_kernel<3, 16>, matmul_tm_kernel<4, 16>, matmul_tm_kernel<7, 16>}};

constexpr uint32_t kMaxParts = 8;

// The grid and the number of planes. A share of the line holds at least one step; with planes, no more than kMaxParts shares touch
// a tile: a tile's steps start within T - c of each other, so that at most (T - c) / share + 2 shares do.
struct TmPlan { uint32_t grid, group_grid, parts, whole, slots, slot_bytes, b_off, group_cost; };
bool tm_plan(const NxTensor *t, int n, uint32_t cols, uint32_t P, bool split, uint32_t groups, int sms, TmPlan &p) {
    const uint32_t nblk = cols / 256;
    uint64_t line = 0, tiles = 0;
    uint32_t raw = 0, longest = 0, cmax = 0;
    for (int i = 0; i < n; ++i) {
        const uint32_t nt = (t[i].rows + kRows - 1) / kRows, c = cost_of(t[i].fmt);
        line += (uint64_t)nt * nblk * c;
        tiles += nt;
        raw = std::max(raw, kRows * pitch_of(t[i].fmt));
        longest = std::max(longest, (nblk - 1) * c);
        cmax = std::max(cmax, c);
    }
    if (line * groups >= (1ull << 31)) return false;
    const uint32_t W = (uint32_t)line, act = (P > 8 ? 16u : 8u) * 1064u;
    p.group_cost = W;
    p.b_off = raw;
    p.slot_bytes = (raw + act + 1023u) & ~1023u;
    p.slots = std::min(kMaxSlots, (kSmemLimit - kHead) / p.slot_bytes);
    p.whole = split ? 0 : 1;
    if (!split) {
        p.group_grid = (uint32_t)std::min<uint64_t>(tiles, 1u << 16);
        p.parts = 1;
    } else {
        uint64_t g = W / cmax;
        if (longest) g = std::min<uint64_t>(g, (uint64_t)W * (kMaxParts - 2) / longest);
        p.group_grid = (uint32_t)std::max<uint64_t>(1, std::min<uint64_t>(g, 1u << 16));
        // one active group: the smallest shares
        const uint32_t one = std::min((uint32_t)sms, p.group_grid);
        p.parts = one == 1 && groups == 1 ? 1 : std::min(kMaxParts, longest / (W / one) + 2);
    }
    p.grid = (uint32_t)std::min<uint64_t>((uint64_t)sms, (uint64_t)p.group_grid * groups);
    return true;
}

} // namespace

cudaError_t matmul_tm_init(void) {
    for (const auto &row : kTmKernels)
        for (auto k : row) {
            const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

uint32_t matmul_tm_parts(const NxTensor *t, int n, uint32_t cols, uint32_t P, bool split, uint32_t groups, int sms) {
    TmPlan p;
    return tm_plan(t, n, cols, P, split, groups, sms, p) ? p.parts : 0;
}

cudaError_t launch_tm_matmul(const NxIn &in, const NxTensor *t, int n, uint32_t cols, uint32_t P, int accumulate, const uint8_t *xq,
                             const uint32_t *xoff, uint32_t *status, int sms, cudaStream_t stream, bool pdl, bool split) {
    TmPlan p;
    const uint32_t groups = in.table ? in.n_groups : 1;
    if (!tm_plan(t, n, cols, P, split, groups, sms, p)) return cudaErrorNotSupported;
    if (accumulate && p.parts > 1) return cudaErrorNotSupported;
    TmArgs k;
    memset(&k, 0, sizeof(k));
    uint32_t fm = 0, base = 0;
    for (int i = 0; i < n; ++i) {
        TmT &d = k.t[i];
        d.y = t[i].y; d.part_stride = t[i].part_stride; d.rows = t[i].rows; d.ystride = t[i].ystride;
        d.tiles = (t[i].rows + kRows - 1) / kRows; d.fmt = t[i].fmt; d.xoff = xoff[i]; d.base = base;
        const uint32_t pitch = t[i].pitch ? t[i].pitch : (uint32_t)row_bytes(t[i].fmt, cols);
        const cudaError_t e = tensor_map_2d(&k.map[i], 8, t[i].w, pitch / 8, (uint64_t)t[i].rows * (in.table ? in.n_experts : 1), pitch,
                                            pitch_of(t[i].fmt) / 8, kRows, false);
        if (e != cudaSuccess) return e;
        base += d.tiles * (cols / 256) * cost_of(t[i].fmt);
        fm |= t[i].fmt == FMT_Q4_K ? 1u : t[i].fmt == FMT_Q6_K ? 2u : 4u;
    }
    k.n = n; k.group_cost = p.group_cost; k.group_grid = p.group_grid; k.nblk = cols / 256; k.P = P; k.parts = p.parts; k.whole = p.whole;
    k.xq = xq; k.accumulate = accumulate; k.rms = in.wnorm ? 1 : 0; k.eps = in.eps;
    k.slots = p.slots; k.slot_bytes = p.slot_bytes; k.b_off = p.b_off;
    k.table = in.table; k.out_idx = in.out_idx; k.list_stride = in.list_stride; k.col_off = in.col_off; k.table_ready = in.table_ready;
    k.status = status;
    const auto kernel = kTmKernels[P > 8 ? 1 : 0][fm == 4 ? 3 : fm > 4 ? 4 : fm - 1];
    return launch_kernel(kernel, dim3(p.grid), dim3(kThreads), kHead + p.slots * p.slot_bytes, stream, pdl, k);
}

} // namespace flb
