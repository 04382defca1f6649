// Several activation columns in one pass over k-quant tensors: Y[p][r] (+)= dot(W[r], X[p]) for p < P <= 16, the
// STREAM_DOT semantics of Task::nx (include/fastllm/fastllm.h:87-96; the reference's GPU form is gdot_i8k_q4_K_mc,
// src/runtime/kernels_gpu.h:682-740, Q4_K only). Used for draft-verification batches, prompt chunks, independent
// sequences and the tokens that share an expert of a mixture-of-experts block. Formats: Q4_K, Q6_K, Q8_0.
//
// A launch is a list of jobs. A job is one tensor (or one expert's slice of it) times one range of columns (a "part":
// one or more segments of 2048 columns whose activation fits in shared memory beside the ring). The items of all jobs
// (a job's units of 16 rows) lie on one line, weighted by their bytes, and every CTA takes an equal, contiguous piece
// of it: one CTA loads the activation of one job, seldom of two. With more than one part the results are partial sums,
// one plane per part, which the next activation conversion (or a small reduce kernel) adds in part order.
//
// Pipeline of a CTA: two groups of 8 consumer warps take the units in turn; each group has its own ring of stages
// (16 rows x one segment, tiled TMA boxes), its own producer warp and its own finalizer warp. Consumer warp w owns the
// 256-column block w of a segment. A warp copies its rows' packed words into registers and releases the stage before it
// computes: two stages per CTA are enough to keep HBM busy, which leaves the shared memory to the activation.
//
// mma.sync m16n8k16: A = 16 rows x 16 weights as f16, the 8 columns of B = 4 tokens as (hi, lo) f16 pairs, NTG
// instructions for 4 NTG tokens from the same A registers.
//   Q4_K : the 6-bit scale of the sub-block goes into A exactly. A masked nibble is, as it stands, the subnormal f16
//          q 2^-24 (q 2^-20 in the high nibble), and one FMA with sc 2^10 (sc 2^6) and -8 sc 2^-14 makes it the f16
//          number (q - 8) sc 2^-14 (|(q - 8) sc| <= 504: exact). A block's 256 columns are then four chains of four
//          instructions, and the super-block scale d is applied once; lane column t unpacks the 32-byte chunk t. The mins
//          and the 8 sc are two more instructions: bf16 (min, scale of sub-block k) times the sub-block sums of the
//          activation as three bf16 parts (24 bits). (q sc instead of (q - 8) sc: larger sums, whose truncation in the
//          tensor core showed.)
//   Q6_K : (q - 32) sc has 13 bits, so the 16 columns of an instruction are one scale group and its f32 result is
//          scaled afterwards (both columns of a pair in one packed FMA).
//   Q8_0 : the same with two instructions per 32-column block and the block's f16 scale.
// Products are exact, sums f32 in a fixed order (warps, then parts): results are reproducible run to run.
//
// What bounds it (B200, 148 SMs): a super-block of 16 rows x 256 columns has to be done in about 100 cycles (Q4_K) to
// keep up with HBM. Tensor pipe: 36 / 72 instructions of 2 cycles per SM for 8 / 16 tokens; shared memory: 8 / 16 KB of
// B per super-block at 128 bytes a cycle; issue: about 400 instructions over four schedulers, which is the bound.
//
// The activations are converted once per call, by a small kernel of their own, into exactly the register image of the
// B operand; the conversion also adds partial sums and a residual, takes SiLU(x) * x2, multiplies by a norm weight (the
// 1 / rms goes onto the results) or adds up the splits of an attention. For the experts of a mixture-of-experts block the
// columns of a job are a device-side list (expert, column count, place of its image): an expert nobody chose costs nothing.
#include "common.cuh"
#include "kernels.h"

#include <cuda_bf16.h>

#include <algorithm>
#include <cstdlib>
#include <cstring>

namespace flb {

namespace {

constexpr int kCW = 8;                                   // consumer warps per group: one per 256-column block of a segment
constexpr uint32_t kConsumers = 2 * kCW;
constexpr uint32_t kThreads = (kConsumers + 4) * 32;     // + two producers, two finalizers
constexpr uint32_t kSeg4 = 8 * 144, kSeg6 = 8 * 210, kSeg8 = 64 * 34;
// Row pitch of a stage in shared memory. Q6_K: 420 words = 4 mod 32, conflict free for lanes (g, t) as it is. Q4_K: 288
// words = 0 mod 32: fetched as 128-byte lines with the 128-byte swizzle (tensor_map_lines_swz), which spreads the same
// 16-byte chunk of 8 consecutive rows over 8 bank groups; rows whose pitch in memory is no multiple of 128 bytes
// (columns no multiple of 2048) use the plain box and pay the conflicts. Q8_0: a segment is wider than a box may be, so
// a stage is two boxes of half a segment, each 16 bytes wider than its half: 276 words = 20 mod 32.
constexpr uint32_t kPitch4 = kSeg4, kPitch6 = kSeg6, kPitch8 = kSeg8 / 2 + 16;
constexpr uint32_t slot_round(uint32_t b) { return (b + 1023u) & ~1023u; }   // the swizzle pattern is tied to the address
constexpr uint32_t kSlot4 = slot_round(16 * kPitch4), kSlot6 = slot_round(16 * kPitch6), kSlot8 = slot_round(32 * kPitch8);
// Image of one 256-column block of a group of four tokens: B fragments, Q4_K: the B operand of the mins, then the
// tokens' power-of-two block scales and the block's sums of squares (RMSNorm).
constexpr uint32_t kFragBytes = 4096, kMinBytes = 256;
constexpr uint32_t kXq4 = kFragBytes + kMinBytes + 32, kXq6 = kFragBytes + 32;
__host__ __device__ constexpr uint32_t xq_bytes(int fmt) { return fmt == FMT_Q4_K ? kXq4 : kXq6; }
__host__ __device__ constexpr uint32_t seg_bytes(int fmt) { return fmt == FMT_Q4_K ? kSeg4 : fmt == FMT_Q6_K ? kSeg6 : kSeg8; }
__host__ __device__ constexpr uint32_t slot_of(int fmt) { return fmt == FMT_Q4_K ? kSlot4 : fmt == FMT_Q6_K ? kSlot6 : kSlot8; }
constexpr uint32_t kSmemLimit = 227 * 1024;
// Shared memory in front: barriers at fixed offsets (full / empty: [2 groups][kMaxSlots]), the CTA's list of pieces, red
// = [2 groups][8 warps][4 NTG tokens][16 rows] f32, the activation, the rings.
constexpr uint32_t kMaxSlots = 12;                       // stages per group
constexpr uint32_t kFull = 0, kEmpty = kFull + 2 * kMaxSlots * 8, kRedFull = kEmpty + 2 * kMaxSlots * 8, kRedEmpty = kRedFull + 16,
                   kXFull = kRedEmpty + 16, kXEmpty = kXFull + 8, kPieces = 512, kBarBytes = 1536;
constexpr uint32_t kMaxPieces = (kBarBytes - kPieces) / 16 - 1;   // word kPieces: their number, the stages per group, the ring's offset; 16 bytes each behind it
static_assert(kXEmpty + 8 <= kPieces, "barriers");

__device__ __forceinline__ uint4 lds128(uint32_t addr) {
    uint4 v;
    asm volatile("ld.shared.v4.u32 {%0, %1, %2, %3}, [%4];" : "=r"(v.x), "=r"(v.y), "=r"(v.z), "=r"(v.w) : "r"(addr));
    return v;
}
__device__ __forceinline__ uint2 lds64(uint32_t addr) {
    uint2 v;
    asm volatile("ld.shared.v2.u32 {%0, %1}, [%2];" : "=r"(v.x), "=r"(v.y) : "r"(addr));
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
__device__ __forceinline__ float ldsf(uint32_t addr) { return __uint_as_float(lds32(addr)); }
__device__ __forceinline__ void sts32(uint32_t addr, float v) { asm volatile("st.shared.f32 [%0], %1;" ::"r"(addr), "f"(v) : "memory"); }
__device__ __forceinline__ uint64_t *bar_at(uint32_t addr) { return reinterpret_cast<uint64_t *>(__cvta_shared_to_generic(addr)); }
__device__ __forceinline__ void bar_arrive(uint32_t bar) {
    asm volatile("mbarrier.arrive.shared::cta.b64 _, [%0];" ::"r"(bar) : "memory");
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
__device__ __forceinline__ bool bar_wait(uint32_t bar, uint32_t parity, uint32_t *status) {
    return bar_try(bar, parity) || mbar_wait_bounded(bar_at(bar), parity, status);
}
// A warp whose wait ran out once waits for nothing any more (its results are void, the status word says so).
__device__ __forceinline__ void bar_wait_or_die(uint32_t bar, uint32_t parity, uint32_t *status, bool &dead) {
    if (dead || bar_try(bar, parity)) return;
    dead = !mbar_wait_bounded(bar_at(bar), parity, status);
}
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
// Byte offset o (a multiple of 16) of a Q4_K row as the stage holds it: as it is, or in the swizzled 128-byte lines.
__device__ __forceinline__ uint32_t q4_row_off(uint32_t o, uint32_t g, bool swz) {
    return swz ? (o & ~127u) + ((((o >> 4) ^ (g + (o >> 7))) & 7u) << 4) : o;
}
__device__ __forceinline__ void mma16816(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                         uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
// The same with a zero accumulator.
__device__ __forceinline__ void mma16816_first(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                               uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.f16.f16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%10, %10, %10, %10};"
                 : "=f"(c[0]), "=f"(c[1]), "=f"(c[2]), "=f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1), "f"(0.f));
}
__device__ __forceinline__ void mma16816_bf16(float (&c)[4], uint32_t a0, uint32_t a1, uint32_t a2, uint32_t a3, uint32_t b0,
                                              uint32_t b1) {
    asm volatile("mma.sync.aligned.m16n8k16.row.col.f32.bf16.bf16.f32 {%0, %1, %2, %3}, {%4, %5, %6, %7}, {%8, %9}, {%0, %1, %2, %3};"
                 : "+f"(c[0]), "+f"(c[1]), "+f"(c[2]), "+f"(c[3])
                 : "r"(a0), "r"(a1), "r"(a2), "r"(a3), "r"(b0), "r"(b1));
}
__device__ __forceinline__ __half2 as_h2(uint32_t v) { return *reinterpret_cast<const __half2 *>(&v); }
__device__ __forceinline__ uint32_t as_u32(__half2 v) { return *reinterpret_cast<const uint32_t *>(&v); }
__device__ __forceinline__ uint32_t hsub2_u32(uint32_t h, __half2 off) { return as_u32(__hsub2(as_h2(h), off)); }
__device__ __forceinline__ uint32_t hfma2_u32(uint32_t h, __half2 m, __half2 c) { return as_u32(__hfma2(as_h2(h), m, c)); }
// the two low bytes (< 64) of w as a pair of bf16 (0x4300 | b is 128 + b)
__device__ __forceinline__ uint32_t bytes_bf16(uint32_t w) {
    const uint32_t b = __byte_perm(w, 0x43434343u, 0x4140u);
    const __nv_bfloat162 v = __hsub2(*reinterpret_cast<const __nv_bfloat162 *>(&b), __floats2bfloat162_rn(128.f, 128.f));
    return *reinterpret_cast<const uint32_t *>(&v);
}
// c + (a, b): both columns of a token in one packed addition
__device__ __forceinline__ float2 add_pair(float2 c, float a, float b) {
    uint64_t cc = *reinterpret_cast<uint64_t *>(&c), ab;
    asm("mov.b64 %0, {%1, %2};" : "=l"(ab) : "f"(a), "f"(b));
    asm("add.rn.f32x2 %0, %0, %1;" : "+l"(cc) : "l"(ab));
    return *reinterpret_cast<float2 *>(&cc);
}
// (c.x, c.y) += s * (a, b): both columns of a token in one packed FMA
__device__ __forceinline__ void fma_pair(float2 &c, float s, float a, float b) {
    uint64_t cc = *reinterpret_cast<uint64_t *>(&c), ss, ab;
    asm("mov.b64 %0, {%1, %1};" : "=l"(ss) : "f"(s));
    asm("mov.b64 %0, {%1, %2};" : "=l"(ab) : "f"(a), "f"(b));
    asm("fma.rn.f32x2 %0, %1, %2, %0;" : "+l"(cc) : "l"(ss), "l"(ab));
    c = *reinterpret_cast<float2 *>(&cc);
}
// byte K of w, which holds s + 128, as the float s (the byte under 0x4B000000 is 2^23 + 128 + s)
__device__ __forceinline__ float s8f(uint32_t w, int k) {
    return __uint_as_float(__byte_perm(w, 0x4B000000u, 0x7440u + k)) - 8388736.f;
}

// ---- activations -> the B operand's register image ----------------------------------------------------------
// An image is [block][token group][xq_bytes]: B fragments of 8 pieces x 32 lanes x 16 bytes, lane = 4 n + t' for column
// n = 2 p' + part (token p' of the group, part 0 = hi, 1 = lo) and lane column t'; a lane's 16 bytes are (b0, b1) of two
// instructions, b0 = columns c + {0, 2}, b1 = c + {1, 3} of its four consecutive columns c ..:
//   Q4_K  piece j    : c = 64 t' + 4 j (low nibbles of word j of chunk t'), then c = 64 t' + 32 + 4 j (high nibbles)
//   Q6_K  piece m / 2: half m & 1, m = (2 hf + hq) * 4 + gq the scale group: c = 128 hf + 32 gq + 16 hq + 4 t'
//   Q8_0  piece b    : c = 32 b + 8 t' + {0, 4}
// Q4_K, then: (b0, b1) per lane of the mins' instruction: b0 = part h of the sums of sub-blocks 2 t', 2 t' + 1, b1 = the
// third part (columns of the lo part) or zero. Then four block scales, four sums of squares.
struct ConvArgs {
    const float *x, *x2;           // column p: row p (or the listed row) of x; x2: the value is SiLU(x) * x2
    size_t part_stride;            // n_parts planes of x (and x2), added in order
    const float *resid;            // + resid (row p, rstride apart)
    float *x_out;                  // the sum is also stored here (row p, rstride apart; may be resid)
    const float *wnorm;            // the value is multiplied by wnorm, the sum of squares of the block recorded
    uint32_t xstride, rstride, n_parts, P, nblk;
    uint8_t *img4, *img6, *img8;   // images wanted (nullptr: not)
    const uint32_t *table, *col_idx;   // grouped columns (see below)
    uint32_t list_stride, col_off, n_groups;   // n_groups: the table has room for so many
    const float *att;              // the columns are attention contexts of heads of 128, added up here from n_splits records
    uint32_t n_splits;             // (attn.cu: [column][head][split][132] = context, maximum, sum)
    int tm;                        // img4 or img6 is the image of matmul_tm.cu
    int dep_first;                 // see NxIn
};
// Device-side table of a grouped launch: word 0 = number of active groups, word 1 = the most token groups of one; then four
// words per active group: {group, number of columns, token groups in front of it, columns in front of it}.

// Four consecutive columns at p, the planes added in order; all of them are requested before the first is used.
__device__ __forceinline__ float4 sum_planes(const float *p, uint32_t n, size_t stride) {
    constexpr int kPlanes = kMaxPlanes;
    static_assert((kNxMaxCols / 256 + 7) / 8 <= kMaxPlanes, "planes of the finest cut, one segment each");
    float4 v[kPlanes];
#pragma unroll
    for (int s = 0; s < kPlanes; ++s) v[s] = (uint32_t)s < n ? *reinterpret_cast<const float4 *>(p + s * stride) : make_float4(0.f, 0.f, 0.f, 0.f);
#pragma unroll
    for (int s = 1; s < kPlanes; ++s) { v[0].x += v[s].x; v[0].y += v[s].y; v[0].z += v[s].z; v[0].w += v[s].w; }
    return v[0];
}

// Four dimensions (4 lane ..) of one head's context from its splits' records (attn_decode_kernel's combine, with all lanes of
// a warp on one head): the weights from every split's maximum and sum, then the contexts in split order, kFlight of them in flight: it is
// bound by the latency of its loads (8 positions, 37 splits, launch to launch: 9.3 us with 16 in flight, three round trips to L2, 5.8 with 40).
template <int kFlight>
__device__ __forceinline__ float4 combine_records(const float *part, uint32_t S, uint32_t lane) {
    const float m0 = lane < S ? __ldcg(part + (size_t)lane * kAttnRecord + 128) : -INFINITY;
    const float m1 = lane + 32 < S ? __ldcg(part + (size_t)(lane + 32) * kAttnRecord + 128) : -INFINITY;
    const float l0 = lane < S ? __ldcg(part + (size_t)lane * kAttnRecord + 129) : 0.f;
    const float l1 = lane + 32 < S ? __ldcg(part + (size_t)(lane + 32) * kAttnRecord + 129) : 0.f;
    float4 acc = make_float4(0.f, 0.f, 0.f, 0.f);
    float w0 = 0.f, w1 = 0.f, L = 1.f;
#pragma unroll 1
    for (uint32_t s0 = 0; s0 < S; s0 += kFlight) {
        float4 ov[kFlight];
#pragma unroll
        for (int j = 0; j < kFlight; ++j)
            ov[j] = s0 + j < S ? __ldcg(reinterpret_cast<const float4 *>(part + (size_t)(s0 + j) * kAttnRecord) + lane) : make_float4(0.f, 0.f, 0.f, 0.f);
        if (s0 == 0) {   // the first contexts are on their way meanwhile
            const float mx = warp_max(fmaxf(m0, m1));
            w0 = m0 == -INFINITY ? 0.f : expf(m0 - mx);
            w1 = m1 == -INFINITY ? 0.f : expf(m1 - mx);
            L = warp_sum(l0 * w0 + l1 * w1);
        }
#pragma unroll
        for (int j = 0; j < kFlight; ++j) {
            const uint32_t sp = s0 + j;
            const float w = __shfl_sync(0xffffffffu, sp < 32 ? w0 : w1, sp & 31u);
            acc.x = fmaf(ov[j].x, w, acc.x); acc.y = fmaf(ov[j].y, w, acc.y);
            acc.z = fmaf(ov[j].z, w, acc.z); acc.w = fmaf(ov[j].w, w, acc.w);
        }
    }
    const float inv = 1.0f / L;
    return make_float4(acc.x * inv, acc.y * inv, acc.z * inv, acc.w * inv);
}

// grid (blocks, columns rounded up to groups of four: grouped, those of all active experts), 64 threads: a block converts 256
// values of one column, a thread four consecutive ones. What bounds it is latency (a launch moves well under a megabyte): hence few
// values per thread, every plane in flight, and as many blocks as there are (block, column) pairs. F: records of a head's splits
// (a.att) in flight, 16 or 40, the latter (254 registers) for those alone. GROUPED: the columns are those of a table. TM: the image is
// that of matmul_tm.cu (8B shape, 8 positions 3110 -> 3088 us, 16 sequences 4432 -> 4392). An instance each,
// since a launch fetches its code from L2 (lookup and records in one instance: passes of the 8B shape 1 % slower). The instance for
// ungrouped columns keeps the records although few launches have any: with them it takes 128 registers, eight blocks an SM; without, 54, and blocks
// that become resident while the matmul in front leaves gather on the first SMs it frees (8 positions, 8 layers of the 8B shape 917 -> 943 us,
// 2048 columns 2.3 % slower). Shared memory reserved for the same eight an SM gives the same time there, but models of 1024 columns in Q8_0 1 to
// 3 % more; the grouped instance, whose launches can be thousands of blocks, does that (launch_nx_convert).
template <int F, bool GROUPED, bool TM>
__global__ void __launch_bounds__(64) act_convert_nx_kernel(const ConvArgs a) {
    __shared__ float2 half_s[2];   // per warp: maximum, sum of squares
    const uint32_t blk = blockIdx.x, warp = threadIdx.x >> 5;
    const uint32_t pp = blockIdx.y & 3u, i = threadIdx.x, hl = i >> 2, tq = i & 3u;   // column of the group; values 16 hl + 4 tq ..
    // launched as a programmatic dependent: the launch itself overlaps the tail of the kernel before, whose output
    // (x, the table) is read only after it has completed
    if (!a.dep_first) griddep_launch_dependents();
    float4 wn = make_float4(1.f, 1.f, 1.f, 1.f);
    if (a.wnorm) wn = __ldg(reinterpret_cast<const float4 *>(a.wnorm + blk * 256 + 4 * i));   // a constant
    griddep_wait();
    if (a.dep_first) griddep_launch_dependents();
    uint32_t n_valid = a.P, tg = blockIdx.y >> 2, ntg = (a.P + 3) / 4, tg0 = 0, grp = 0, row0 = 0;
    if (GROUPED) {   // the group of four is one of all active experts' together: look its expert up
        const uint32_t n_act = a.table[0], lane = threadIdx.x & 31u, at = tg;
        ntg = 0;
        for (uint32_t b = 0; b < a.n_groups && ntg == 0; b += 32) {
            uint4 e = make_uint4(0u, 0u, 0u, 0u);
            if (b + lane < a.n_groups) e = reinterpret_cast<const uint4 *>(a.table)[1 + b + lane];   // requested together with n_act
            if (b + lane >= n_act) e.y = 0;
            const uint32_t n = (e.y + 3) / 4, mask = __ballot_sync(0xffffffffu, at - e.z < n);
            if (mask) {
                const int l = __ffs(mask) - 1;
                grp = __shfl_sync(0xffffffffu, e.x, l); n_valid = __shfl_sync(0xffffffffu, e.y, l);
                tg0 = __shfl_sync(0xffffffffu, e.z, l); row0 = __shfl_sync(0xffffffffu, e.w, l);
                ntg = __shfl_sync(0xffffffffu, n, l);
            }
        }
        if (ntg == 0) return;
        tg = at - tg0;
    }
    const uint32_t p = 4 * tg + pp;
    float4 v = make_float4(0.f, 0.f, 0.f, 0.f);
    float ss = 0.f;
    if (p < n_valid) {
        const size_t row = GROUPED && a.col_idx ? a.col_idx[(size_t)grp * a.list_stride + a.col_off + p] : row0 + p;
        const size_t at = row * a.xstride + blk * 256 + 4 * i, rat = (size_t)p * a.rstride + blk * 256 + 4 * i;
        float4 r = make_float4(0.f, 0.f, 0.f, 0.f);
        if (a.resid) r = *reinterpret_cast<const float4 *>(a.resid + rat);
        if (!GROUPED && a.att) v = combine_records<F>(a.att + ((size_t)p * (2 * a.nblk) + 2 * blk + warp) * a.n_splits * kAttnRecord, a.n_splits, threadIdx.x & 31u);
        else v = sum_planes(a.x + at, a.n_parts, a.part_stride);
        if (a.x2) {   // fl_op_silu_mul (src/runtime/decode_params.h:267-272)
            const float4 u = sum_planes(a.x2 + at, a.n_parts, a.part_stride);
            v.x = (v.x / (1.0f + expf(-v.x))) * u.x; v.y = (v.y / (1.0f + expf(-v.y))) * u.y;
            v.z = (v.z / (1.0f + expf(-v.z))) * u.z; v.w = (v.w / (1.0f + expf(-v.w))) * u.w;
        }
        if (a.resid) { v.x += r.x; v.y += r.y; v.z += r.z; v.w += r.w; }
        if (a.x_out) *reinterpret_cast<float4 *>(a.x_out + rat) = v;
        if (a.wnorm) {
            ss = (v.x * v.x + v.y * v.y) + (v.z * v.z + v.w * v.w);
            v.x *= wn.x; v.y *= wn.y; v.z *= wn.z; v.w *= wn.w;
        }
    }
    if (!a.img4 && !a.img6 && !a.img8) return;   // only the sum was asked for
    float amax = fmaxf(fmaxf(fabsf(v.x), fabsf(v.y)), fmaxf(fabsf(v.z), fabsf(v.w)));
    amax = warp_max(amax);
    ss = warp_sum(ss);
    if ((threadIdx.x & 31u) == 0) half_s[warp] = make_float2(amax, ss);
    __syncthreads();
    const float2 h0 = half_s[0], h1 = half_s[1];
    amax = fmaxf(h0.x, h1.x);
    // block scale 2^e with amax / 2^e in [2^13, 2^14); e clamped so that both 2^e and 2^-e are normal floats
    int e = (int)((__float_as_uint(amax) >> 23) & 0xFFu) - 127 - 13;
    e = amax > 0.f ? max(-126, min(e, 114)) : 0;
    const float inv_s = __uint_as_float((uint32_t)(127 - e) << 23), scale = __uint_as_float((uint32_t)(127 + e) << 23);
    const float s0 = v.x * inv_s, s1 = v.y * inv_s, s2 = v.z * inv_s, s3 = v.w * inv_s;
    const __half2 h02 = __floats2half2_rn(s0, s2), h13 = __floats2half2_rn(s1, s3);
    const float2 f02 = __half22float2(h02), f13 = __half22float2(h13);
    const __half2 l02 = __floats2half2_rn(s0 - f02.x, s2 - f02.y), l13 = __floats2half2_rn(s1 - f13.x, s3 - f13.y);
    const float2 g02 = __half22float2(l02), g13 = __half22float2(l13);
    const uint2 hi = make_uint2(as_u32(h02), as_u32(h13)), lo = make_uint2(as_u32(l02), as_u32(l13));
    float sum = ((f02.x + g02.x) + (f13.x + g13.x)) + ((f02.y + g02.y) + (f13.y + g13.y));
#pragma unroll
    for (int o = 1; o < 8; o <<= 1) sum += __shfl_xor_sync(0xffffffffu, sum, o);   // over the 32-column sub-block
    if (TM) {
        // Image of a block for NT = 8 or 16 tokens (matmul_tm.cu): a tile per 64 columns of 2 NT rows of 128 bytes (row p the hi parts
        // of token p, row NT + p the lo parts; 16-byte piece j of a row at j ^ (row & 7), the 128-byte swizzle), then the
        // sub-block sums [8][NT], the block scales [NT] and the sums of squares [NT]. Q4_K, piece j: columns 4 j + {0, 2, 1, 3} of
        // the first sub-block of the tile, then of the second. Q6_K, tile 2 hf + hq, pieces 2 gq and 2 gq + 1: columns c, c + 2
        // and c + 1, c + 3 for c = 128 hf + 32 gq + 16 hq + 4 t, t = 0 .. 3. Rows of tokens that there are not are never written
        // nor used.
        if (p >= n_valid) return;
        const uint32_t NT = n_valid > 8 ? 16u : 8u;
        uint8_t *img = (a.img4 ? a.img4 : a.img6) + (size_t)blk * (NT * 1064u);
        // (NT is a multiple of 8: the rows of both parts swizzle alike)
        if (a.img4) {
            uint8_t *row = img + (i >> 4) * (NT * 256) + p * 128 + (((i & 7u) ^ (p & 7u)) << 4) + (i & 8u);
            *reinterpret_cast<uint2 *>(row) = hi;
            *reinterpret_cast<uint2 *>(row + NT * 128) = lo;
        } else {
            uint8_t *row = img + ((i >> 5) * 2 + ((i >> 2) & 1u)) * (NT * 256) + p * 128 + 4 * (i & 3u);
            const uint32_t j = 2 * ((i >> 3) & 3u), j0 = (j ^ (p & 7u)) << 4, j1 = ((j + 1) ^ (p & 7u)) << 4;
            *reinterpret_cast<uint32_t *>(row + j0) = hi.x;
            *reinterpret_cast<uint32_t *>(row + j1) = hi.y;
            *reinterpret_cast<uint32_t *>(row + NT * 128 + j0) = lo.x;
            *reinterpret_cast<uint32_t *>(row + NT * 128 + j1) = lo.y;
        }
        float *side = reinterpret_cast<float *>(img + NT * 1024);
        if ((i & 7u) == 0) side[(i >> 3) * NT + p] = sum;
        if (i == 0) { side[8 * NT + p] = scale; side[9 * NT + p] = h0.y + h1.y; }
        return;
    }
    const size_t unit = (size_t)tg0 * a.nblk + (size_t)blk * ntg + tg;
#pragma unroll
    for (int f = 0; f < 3; ++f) {
        uint8_t *base = f == 0 ? a.img4 : f == 1 ? a.img6 : a.img8;
        if (!base) continue;
        base += unit * (f == 0 ? kXq4 : kXq6);
        uint32_t off, t;   // byte offset but for the lane, lane column
        if (f == 0) {
            off = (4 * (hl & 1u) + tq) * 512u + ((hl >> 1) & 1u) * 8u; t = hl >> 2;
        } else if (f == 1) {
            const uint32_t m = (((hl >> 3) * 2 + (hl & 1u)) * 4) + ((hl >> 1) & 3u);
            off = (m >> 1) * 512u + (m & 1u) * 8u; t = tq;
        } else {
            off = (hl >> 1) * 512u + (tq & 1) * 8u; t = 2 * (hl & 1u) + (tq >> 1);
        }
        *reinterpret_cast<uint2 *>(base + off + (4 * (2 * pp) + t) * 16u) = hi;
        *reinterpret_cast<uint2 *>(base + off + (4 * (2 * pp + 1) + t) * 16u) = lo;
        uint8_t *tail = base + kFragBytes;
        if (f == 0) {
            if ((i & 7u) == 0) {   // the sum of sub-block sb in three bf16 parts (exact: 24 bits)
                const uint32_t sb = i >> 3;
                const __nv_bfloat16 p0 = __float2bfloat16_rn(sum);
                const float r1 = sum - __bfloat162float(p0);
                const __nv_bfloat16 p1 = __float2bfloat16_rn(r1);
                const __nv_bfloat16 p2 = __float2bfloat16_rn(r1 - __bfloat162float(p1));
                uint8_t *d0 = tail + (4 * (2 * pp) + (sb >> 1)) * 8u + (sb & 1u) * 2u;
                uint8_t *d1 = tail + (4 * (2 * pp + 1) + (sb >> 1)) * 8u + (sb & 1u) * 2u;
                *reinterpret_cast<__nv_bfloat16 *>(d0) = p0;
                *reinterpret_cast<uint16_t *>(d0 + 4) = 0;
                *reinterpret_cast<__nv_bfloat16 *>(d1) = p1;
                *reinterpret_cast<__nv_bfloat16 *>(d1 + 4) = p2;
            }
            tail += kMinBytes;
        }
        if (i == 0) {
            reinterpret_cast<float *>(tail)[pp] = scale;
            reinterpret_cast<float *>(tail)[4 + pp] = h0.y + h1.y;
        }
    }
}

// y[p][r] (+)= sum over the parts of part[s][p][r]
__global__ void __launch_bounds__(256) reduce_parts_kernel(const float *__restrict__ part, size_t part_stride, uint32_t n_parts,
                                                           float *y, uint32_t rows, uint32_t ystride, int accumulate) {
    griddep_launch_dependents();
    griddep_wait();
    const uint32_t r = blockIdx.x * 256 + threadIdx.x, p = blockIdx.y;
    if (r >= rows) return;
    float v = 0.f;
#pragma unroll 4
    for (uint32_t s = 0; s < n_parts; ++s) v += part[s * part_stride + (size_t)p * rows + r];
    float *dst = y + (size_t)p * ystride + r;
    *dst = accumulate ? *dst + v : v;
}

struct NxT {
    float *y;
    size_t part_stride;            // floats between the planes of the parts
    uint32_t rows, ystride, units, xoff;   // xoff: bytes from xq to the image of this format
    int fmt, swz;
};
struct NxJob { uint32_t base, cost; uint16_t tensor, part, seg0, nseg; };   // base: where the job starts on the line of a group
constexpr int kMaxJobs = 32;

struct NxArgs {
    CUtensorMap map[3];            // the tiled views a stage's boxes are cut from
    NxT t[3];
    NxJob job[kMaxJobs];
    uint32_t n_jobs, group_cost, nblk, P;
    const uint8_t *xq;
    int accumulate, rms;
    float eps;
    uint32_t slot_bytes, x_off, x_blk_tg;   // x_blk_tg: bytes of a part's activation per token group
    uint32_t red_group;            // floats between the groups' reduction buffers (for the widest piece of the launch)
    // grouped launches: active groups from the table, output rows from the list (or numbered through)
    const uint32_t *table, *out_idx;
    uint32_t list_stride, col_off;
    int table_ready;               // the table was complete before the previous kernel started
    uint32_t *status;
};

__host__ __device__ constexpr uint32_t nx_ring_off(uint32_t x_off, uint32_t x_blk_tg, uint32_t ntg) {
    return (x_off + x_blk_tg * ntg + 1023u) & ~1023u;
}

// The pieces of this CTA, listed in shared memory by one thread at the start: {first unit, last unit, job | columns << 8 |
// group << 16, columns in front << 16 | token groups in front << 2 | same activation as the piece before << 1 | parity of the
// units before}.
struct NxPiece { uint32_t u0, u1, job, n_valid, grp, row0, tg0, same, par; };
__device__ __forceinline__ NxPiece nx_piece(uint32_t smem, uint32_t i) {
    const uint4 v = lds128(smem + kPieces + 16 + 16 * i);
    return NxPiece{v.x, v.y, v.z & 0xFFu, (v.z >> 8) & 0xFFu, v.z >> 16, v.w >> 16, (v.w >> 2) & 0x3FFFu, (v.w >> 1) & 1u, v.w & 1u};
}
__device__ __noinline__ void nx_list_pieces(const NxArgs &a, uint8_t *smem_raw) {
    uint32_t *count = reinterpret_cast<uint32_t *>(smem_raw + kPieces);
    uint4 *out = reinterpret_cast<uint4 *>(smem_raw + kPieces + 16);
    uint32_t n = 0, kk = 0, last_g = 0, last_part = 0, last_x = 0;
    const uint32_t n_act = a.table ? a.table[0] : 1u;
    // the activation region is as large as the widest piece of this launch needs (grouped: known here only), the ring has the rest
    const uint32_t ring_off = nx_ring_off(a.x_off, a.x_blk_tg, a.table ? a.table[1] : (a.P + 3) / 4);
    count[1] = min((kSmemLimit - ring_off) / (2 * a.slot_bytes), kMaxSlots);
    count[2] = ring_off;
    const uint32_t W = a.group_cost * n_act;   // < 2^31 (checked on the host)
    const uint32_t wq = W / gridDim.x, wr = W % gridDim.x;   // equal shares, W x / gridDim.x without 64-bit divisions
    const uint32_t lo = wq * blockIdx.x + wr * blockIdx.x / gridDim.x, hi = wq * (blockIdx.x + 1) + wr * (blockIdx.x + 1) / gridDim.x;
    for (uint32_t g = lo / a.group_cost; g < n_act && g * a.group_cost < hi; ++g) {
        uint4 e = make_uint4(0u, a.P, 0u, 0u);
        if (a.table) e = reinterpret_cast<const uint4 *>(a.table)[1 + g];
        for (uint32_t j = 0; j < a.n_jobs && n < kMaxPieces; ++j) {
            const NxJob &jb = a.job[j];
            const uint32_t units = a.t[jb.tensor].units, b = g * a.group_cost + jb.base, end = b + units * jb.cost;
            if (end <= lo || b >= hi) continue;
            const uint32_t u0 = b >= lo ? 0u : (lo - b + jb.cost - 1) / jb.cost;
            const uint32_t u1 = end <= hi ? units : (hi - b + jb.cost - 1) / jb.cost;
            if (u0 >= u1) continue;
            const uint32_t same = n > 0 && last_g == g && last_part == jb.part && last_x == a.t[jb.tensor].xoff ? 1u : 0u;
            last_g = g; last_part = jb.part; last_x = a.t[jb.tensor].xoff;
            out[n++] = make_uint4(u0, u1, j | (e.y << 8) | (e.x << 16), (e.w << 16) | (e.z << 2) | (same << 1) | (kk & 1u));
            kk += u1 - u0;
        }
    }
    *count = n;
}

// ---- per-block math: rows g (row 0) and g + 8 (row 1), tokens 4 tg + t ---------------------------------------------
// acc[row][tg] += the block's contribution. `release` runs after the last read of the stage. offs: where the block's
// header and the two halves of chunk t lie in a row, in 16 bytes, one byte each.
template <int NTG, typename Rel>
__device__ __forceinline__ void q4k_block_nx(uint32_t r0, uint32_t offs, uint32_t t, uint32_t xaddr, uint32_t lane, float (&acc)[2][NTG],
                                             Rel &&release) {
    const uint32_t r1 = r0 + 8 * kPitch4, oh = (offs & 0xFFu) * 16u, oa = ((offs >> 8) & 0xFFu) * 16u, ob = (offs >> 16) * 16u;
    uint4 wa[2], wb[2], hd[2];
    wa[0] = lds128(r0 + oa); wa[1] = lds128(r1 + oa);
    hd[0] = lds128(r0 + oh); hd[1] = lds128(r1 + oh);
    wb[0] = lds128(r0 + ob); wb[1] = lds128(r1 + ob);
    release();
    // 6-bit scales / mins of sub-blocks 2t, 2t+1 (packing: fl_q4k_scale_min, src/runtime/quants.h:121-129): sub-blocks
    // 0..3 are the low six bits of bytes 0..3 (4..7 for the mins), 4..7 a nibble of bytes 8..11 under the top two bits of those
    const uint32_t sh = 16u * (t & 1u);
    const uint32_t shA = t >= 2 ? sh + 2u : sh, mA = t >= 2 ? 0x3030u : 0x3F3Fu, mE = t >= 2 ? 0x0F0Fu : 0u;
    __half2 sL[2], sH[2], kL[2], kH[2];   // scales times 2^10 (low nibbles), 2^6 (high nibbles); -8 2^-14 times the scales
    uint32_t sm[2];                       // the two sub-blocks' scales and mins, a byte each
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t sc = ((hd[r].y >> shA) & mA) | ((hd[r].w >> sh) & mE);
        const uint32_t mn = ((hd[r].z >> shA) & mA) | ((hd[r].w >> (sh + 4u)) & mE);
        const __half2 k1024 = __floats2half2_rn(1024.f, 1024.f);
        const __half2 s0 = __hsub2(as_h2(__byte_perm(sc, 0x64646464u, 0x4040u)), k1024), s1 = __hsub2(as_h2(__byte_perm(sc, 0x64646464u, 0x4141u)), k1024);
        const __half2 km8 = __floats2half2_rn(-0.00048828125f, -0.00048828125f);   // -8 2^-14
        sL[r] = __hmul2(s0, k1024); kL[r] = __hmul2(s0, km8);
        sH[r] = __hmul2(s1, __floats2half2_rn(64.f, 64.f)); kH[r] = __hmul2(s1, km8);
        sm[r] = sc | (mn << 16);
    }
    // The tensor core truncates its running sum at every instruction, always towards zero: an error that grows with the length
    // of a chain and has the sum's own sign, so that it does not average out over blocks and adds up over the matmuls of a
    // layer (chains of 8: -1.0e-7 of every result; a block of experts 4.8e-7 off, of 4 as here 3.1e-7, a scale group at a time,
    // the form before, 4.1e-7). Hence chains of 4 from zero, added with rounding. Up to 8 tokens (NTG <= 2) all four chains of a
    // block side by side, added at the end, both columns of a token (hi, lo) at once: the additions wait for nothing (14336 x
    // 4096, 4 tokens: 17.1 us as with chains of 8; added half-way 18.5). Else one at a time, their sums put aside: the
    // registers of two do not fit (16 tokens: 30.0 against 28.9 us).
    constexpr bool kSide = NTG <= 2;
    constexpr int kStep = kSide ? 4 : 2;   // words (two instructions each) between two chains
    float c[kSide ? 4 : 1][NTG][4], sum[2][NTG];
    const uint32_t ML = 0x000F000Fu, MH = 0x00F000F0u;
#pragma unroll
    for (int j = 0; j < 8; ++j) {
        const uint4 &q0 = j < 4 ? wa[0] : wb[0], &q1 = j < 4 ? wa[1] : wb[1];
        const uint32_t W0 = (j & 3) == 0 ? q0.x : (j & 3) == 1 ? q0.y : (j & 3) == 2 ? q0.z : q0.w;
        const uint32_t W1 = (j & 3) == 0 ? q1.x : (j & 3) == 1 ? q1.y : (j & 3) == 2 ? q1.z : q1.w;
        const uint32_t V0 = W0 >> 8, V1 = W1 >> 8;
        const uint32_t l0 = hfma2_u32(W0 & ML, sL[0], kL[0]), l1 = hfma2_u32(W1 & ML, sL[1], kL[1]);
        const uint32_t l2 = hfma2_u32(V0 & ML, sL[0], kL[0]), l3 = hfma2_u32(V1 & ML, sL[1], kL[1]);
        const uint32_t h0 = hfma2_u32(W0 & MH, sH[0], kH[0]), h1 = hfma2_u32(W1 & MH, sH[1], kH[1]);
        const uint32_t h2 = hfma2_u32(V0 & MH, sH[0], kH[0]), h3 = hfma2_u32(V1 & MH, sH[1], kH[1]);
        const int lo = kSide ? j / kStep * 2 : 0, hi = kSide ? lo + 1 : 0;   // the chains of the low and of the high nibbles
#pragma unroll
        for (int tg = 0; tg < NTG; ++tg) {
            const uint4 b = lds128(xaddr + tg * kXq4 + j * 512 + lane * 16);
            if (j % kStep == 0) mma16816_first(c[lo][tg], l0, l1, l2, l3, b.x, b.y);
            else mma16816(c[lo][tg], l0, l1, l2, l3, b.x, b.y);
            if (kSide && j % kStep == 0) mma16816_first(c[hi][tg], h0, h1, h2, h3, b.z, b.w);
            else mma16816(c[hi][tg], h0, h1, h2, h3, b.z, b.w);
        }
        if (!kSide && j % kStep == kStep - 1)
#pragma unroll
            for (int tg = 0; tg < NTG; ++tg)
#pragma unroll
                for (int r = 0; r < 2; ++r) {
                    const float v = c[0][tg][2 * r] + c[0][tg][2 * r + 1];
                    sum[r][tg] = j < kStep ? v : sum[r][tg] + v;
                }
    }
    if (kSide)
#pragma unroll
        for (int tg = 0; tg < NTG; ++tg)
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                float2 v = make_float2(c[0][tg][2 * r], c[0][tg][2 * r + 1]);
#pragma unroll
                for (int i = 1; i < (kSide ? 4 : 1); ++i) v = add_pair(v, c[i][tg][2 * r], c[i][tg][2 * r + 1]);
                sum[r][tg] = v.x + v.y;
            }
    const float d0 = h2f_bits((uint16_t)(hd[0].x & 0xFFFFu)), e0 = h2f_bits((uint16_t)(hd[0].x >> 16));
    const uint32_t as[2] = {bytes_bf16(sm[0]), bytes_bf16(sm[1])}, am[2] = {bytes_bf16(sm[0] >> 16), bytes_bf16(sm[1] >> 16)};
    const float d1 = h2f_bits((uint16_t)(hd[1].x & 0xFFFFu)), e1 = h2f_bits((uint16_t)(hd[1].x >> 16));
#pragma unroll
    for (int tg = 0; tg < NTG; ++tg) {
        float m[4] = {0.f, 0.f, 0.f, 0.f}, s[4] = {0.f, 0.f, 0.f, 0.f};
        const uint2 b = lds64(xaddr + tg * kXq4 + kFragBytes + lane * 8);
        mma16816_bf16(m, am[0], am[1], am[0], am[1], b.x, b.y);
        mma16816_bf16(s, as[0], as[1], as[0], as[1], b.x, b.y);
        const float xs = ldsf(xaddr + tg * kXq4 + kFragBytes + kMinBytes + t * 4);
        // 8 d (s) - e (m) is mostly a difference of nearly equal numbers (a min is about 8 steps of the scale): the sums over the
        // leading parts, s[0] and m[0], carry at most 24 bits, so that theirs is formed first, without rounding the product
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float d = r ? d1 : d0, e = r ? e1 : e0, p = __fmul_rn(e, m[2 * r]);
            float v = fmaf(8.f * d, s[2 * r], -p) - fmaf(e, m[2 * r], -p);
            v = fmaf(-e, m[2 * r + 1], fmaf(8.f * d, s[2 * r + 1], v));
            acc[r][tg] = fmaf(xs, fmaf(16384.f * d, sum[r][tg], v), acc[r][tg]);
        }
    }
}

// Q6_K (q = nibble | two high bits << 4, value d * sc * (q - 32); fl_dot_row_q6_K, src/runtime/quants.h:194-230): an
// instruction covers the 16 columns of one int8 scale; lane column t unpacks bytes 4 t .. 4 t + 3 of the 16-byte runs.
// ODD: the block starts 2 bytes past a word boundary (r0 is the aligned address 2 bytes in front of it).
template <int NTG, bool ODD, typename Rel>
__device__ __forceinline__ void q6k_block_nx(uint32_t r0, uint32_t t, uint32_t xaddr, uint32_t lane, float (&acc)[2][NTG], Rel &&release) {
    uint32_t wa[2][4], wb[2][4], wh[2][4];   // [row][(hf, hq)]
    uint32_t sw[2][4];                       // the 16 int8 scales as (s + 128) bytes
    float dd[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t rb = r0 + r * 8 * kPitch6;
#pragma unroll
        for (int hh = 0; hh < 4; ++hh) {
            const uint32_t hf = hh >> 1, hq = hh & 1;
            const uint32_t oa = 64 * hf + 16 * hq + 4 * t, oh = 128 + 32 * hf + 16 * hq + 4 * t;
            if (ODD) {
                wa[r][hh] = __byte_perm(lds32(rb + oa), lds32(rb + oa + 4), 0x5432u);
                wb[r][hh] = __byte_perm(lds32(rb + oa + 32), lds32(rb + oa + 36), 0x5432u);
                wh[r][hh] = __byte_perm(lds32(rb + oh), lds32(rb + oh + 4), 0x5432u);
            } else {
                wa[r][hh] = lds32(rb + oa);
                wb[r][hh] = lds32(rb + oa + 32);
                wh[r][hh] = lds32(rb + oh);
            }
        }
        if (ODD) {
            uint32_t s[5];
#pragma unroll
            for (int k = 0; k < 5; ++k) s[k] = lds32(rb + 192 + 4 * k);
#pragma unroll
            for (int k = 0; k < 4; ++k) sw[r][k] = __byte_perm(s[k], s[k + 1], 0x5432u) ^ 0x80808080u;
            dd[r] = h2f_bits((uint16_t)(lds32(rb + 208) >> 16));
        } else {
#pragma unroll
            for (int k = 0; k < 4; ++k) sw[r][k] = lds32(rb + 192 + 4 * k) ^ 0x80808080u;
            dd[r] = h2f_bits((uint16_t)lds16(rb + 208));
        }
    }
    release();
    float2 s2[2][NTG];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int tg = 0; tg < NTG; ++tg) s2[r][tg] = make_float2(0.f, 0.f);
    const __half2 off = __floats2half2_rn(1056.f, 1056.f);
#pragma unroll
    for (int hh = 0; hh < 4; ++hh) {
        const int hf = hh >> 1, hq = hh & 1;
        uint32_t q[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t a = wa[r][hh], b = wb[r][hh], h = wh[r][hh];
            q[r][0] = (a & 0x0F0F0F0Fu) | ((h << 4) & 0x30303030u);
            q[r][1] = (b & 0x0F0F0F0Fu) | ((h << 2) & 0x30303030u);
            q[r][2] = ((a >> 4) & 0x0F0F0F0Fu) | (h & 0x30303030u);
            q[r][3] = ((b >> 4) & 0x0F0F0F0Fu) | ((h >> 2) & 0x30303030u);
        }
#pragma unroll
        for (int gp = 0; gp < 2; ++gp) {   // groups 2 gp, 2 gp + 1: one 16-byte piece of B
            float c[2][NTG][4];
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int gq = 2 * gp + i;
                // bytes 0, 2 / 1, 3 under 0x64: f16 1024 + q; minus 1056 is q - 32, exact
                const uint32_t a0 = hsub2_u32(__byte_perm(q[0][gq], 0x64646464u, 0x4240u), off), a1 = hsub2_u32(__byte_perm(q[1][gq], 0x64646464u, 0x4240u), off);
                const uint32_t a2 = hsub2_u32(__byte_perm(q[0][gq], 0x64646464u, 0x4341u), off), a3 = hsub2_u32(__byte_perm(q[1][gq], 0x64646464u, 0x4341u), off);
#pragma unroll
                for (int tg = 0; tg < NTG; ++tg) {
                    const uint2 b = lds64(xaddr + tg * kXq6 + (hh * 2 + gp) * 512 + lane * 16 + i * 8);
                    c[i][tg][0] = c[i][tg][1] = c[i][tg][2] = c[i][tg][3] = 0.f;
                    mma16816(c[i][tg], a0, a1, a2, a3, b.x, b.y);
                }
            }
#pragma unroll
            for (int i = 0; i < 2; ++i) {
                const int si = 8 * hf + 2 * (2 * gp + i) + hq;
                const float f0 = s8f(sw[0][si >> 2], si & 3), f1 = s8f(sw[1][si >> 2], si & 3);
#pragma unroll
                for (int tg = 0; tg < NTG; ++tg) {
                    fma_pair(s2[0][tg], f0, c[i][tg][0], c[i][tg][1]);
                    fma_pair(s2[1][tg], f1, c[i][tg][2], c[i][tg][3]);
                }
            }
        }
    }
#pragma unroll
    for (int tg = 0; tg < NTG; ++tg) {
        const float xs = ldsf(xaddr + tg * kXq6 + kFragBytes + t * 4);
        acc[0][tg] = fmaf(xs, dd[0] * (s2[0][tg].x + s2[0][tg].y), acc[0][tg]);
        acc[1][tg] = fmaf(xs, dd[1] * (s2[1][tg].x + s2[1][tg].y), acc[1][tg]);
    }
}

// Q8_0 (blocks of 32 int8 with one f16 d, 34 bytes; fl_dot_row_q8_0, src/runtime/quants.h:132-142): lane column t takes
// bytes 8 t .. 8 t + 7 of a block, two instructions per block. Even blocks start on a word boundary, so their quants
// are 2 bytes past one; odd blocks' quants are aligned. An int8 s becomes f16 through (s ^ 0x80) under 0x64: 1024 + 128 + s.
template <int NTG, typename Rel>
__device__ __forceinline__ void q80_block_nx(uint32_t r0, uint32_t t, uint32_t xaddr, uint32_t lane, float (&acc)[2][NTG], Rel &&release) {
    uint32_t w[2][8][2];
    uint32_t dw[2][4];   // scales of blocks 2 b, 2 b + 1 as a pair of halves
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t rb = r0 + r * 8 * kPitch8;
#pragma unroll
        for (int b = 0; b < 4; ++b) {   // pairs of blocks: 68 bytes
            const uint32_t p = rb + 68 * b, q = p + 8 * t;
            const uint32_t x0 = lds32(q), x1 = lds32(q + 4), x2 = lds32(q + 8);
            w[r][2 * b][0] = __byte_perm(x0, x1, 0x5432u) ^ 0x80808080u;
            w[r][2 * b][1] = __byte_perm(x1, x2, 0x5432u) ^ 0x80808080u;
            w[r][2 * b + 1][0] = lds32(q + 36) ^ 0x80808080u;
            w[r][2 * b + 1][1] = lds32(q + 40) ^ 0x80808080u;
            dw[r][b] = lds16(p) | (lds32(p + 32) & 0xFFFF0000u);
        }
    }
    release();
    float2 s2[2][NTG];
#pragma unroll
    for (int r = 0; r < 2; ++r)
#pragma unroll
        for (int tg = 0; tg < NTG; ++tg) s2[r][tg] = make_float2(0.f, 0.f);
    const __half2 off = __floats2half2_rn(1152.f, 1152.f);
#pragma unroll
    for (int b = 0; b < 8; ++b) {
        uint32_t a[2][4];
#pragma unroll
        for (int i = 0; i < 2; ++i) {
            a[i][0] = hsub2_u32(__byte_perm(w[0][b][i], 0x64646464u, 0x4240u), off);
            a[i][1] = hsub2_u32(__byte_perm(w[1][b][i], 0x64646464u, 0x4240u), off);
            a[i][2] = hsub2_u32(__byte_perm(w[0][b][i], 0x64646464u, 0x4341u), off);
            a[i][3] = hsub2_u32(__byte_perm(w[1][b][i], 0x64646464u, 0x4341u), off);
        }
        const uint32_t h0 = dw[0][b >> 1], h1 = dw[1][b >> 1];
        const float f0 = h2f_bits((uint16_t)((b & 1) ? h0 >> 16 : h0 & 0xFFFFu)), f1 = h2f_bits((uint16_t)((b & 1) ? h1 >> 16 : h1 & 0xFFFFu));
#pragma unroll
        for (int tg = 0; tg < NTG; ++tg) {
            const uint4 x = lds128(xaddr + tg * kXq6 + b * 512 + lane * 16);
            float c[4] = {0.f, 0.f, 0.f, 0.f};
            mma16816(c, a[0][0], a[0][1], a[0][2], a[0][3], x.x, x.y);
            mma16816(c, a[1][0], a[1][1], a[1][2], a[1][3], x.z, x.w);
            fma_pair(s2[0][tg], f0, c[0], c[1]);
            fma_pair(s2[1][tg], f1, c[2], c[3]);
        }
    }
#pragma unroll
    for (int tg = 0; tg < NTG; ++tg) {
        const float xs = ldsf(xaddr + tg * kXq6 + kFragBytes + t * 4);
        acc[0][tg] = fmaf(xs, s2[0][tg].x + s2[0][tg].y, acc[0][tg]);
        acc[1][tg] = fmaf(xs, s2[1][tg].x + s2[1][tg].y, acc[1][tg]);
    }
}

struct NxRing { uint32_t slot, par, slots, base; };   // a group's next stage and its parity, carried from piece to piece; its ring

// One consumer warp's share of a piece: units u0, u0 + 2, ... of format FMT with NTG token groups.
template <int FMT, int NTG>
__device__ __forceinline__ void consume(const NxArgs &a, uint32_t smem, const NxJob &jb, uint32_t u0, uint32_t u1, uint32_t grp8,
                                        uint32_t w, uint32_t lane, NxRing &rg, uint32_t &red_par, bool &dead) {
    const uint32_t xs_addr = smem + a.x_off;
    const uint32_t g = lane >> 2, t = lane & 3u;
    const uint32_t nblk_p = min(a.nblk - jb.seg0 * 8u, jb.nseg * 8u);   // blocks of the part
    const bool swz = FMT == FMT_Q4_K && a.t[jb.tensor].swz != 0;
    uint32_t offs = 0;   // see q4k_block_nx
    if (FMT == FMT_Q4_K)
        offs = (q4_row_off(w * 144u, g, swz) >> 4) | (q4_row_off(w * 144u + 16u + 32u * t, g, swz) << 4) |
               (q4_row_off(w * 144u + 32u + 32u * t, g, swz) << 12);
    for (uint32_t u = u0; u < u1; u += 2) {
        float acc[2][NTG];
#pragma unroll
        for (int tg = 0; tg < NTG; ++tg) acc[0][tg] = acc[1][tg] = 0.f;
#pragma unroll 1
        for (uint32_t seg = 0; seg < jb.nseg; ++seg) {
            const uint32_t blk = seg * 8 + w, bar = smem + (grp8 * kMaxSlots + rg.slot) * 8;
            bar_wait_or_die(bar + kFull, rg.par, a.status, dead);
            auto release = [&]() {
                __syncwarp();
                if (lane == 0) bar_arrive(bar + kEmpty);
            };
            const uint32_t st = rg.base + rg.slot * a.slot_bytes, xaddr = xs_addr + blk * (NTG * xq_bytes(FMT));
            if (blk >= nblk_p) release();
            else if (FMT == FMT_Q4_K) q4k_block_nx<NTG>(st + g * kPitch4, offs, t, xaddr, lane, acc, release);
            else if (FMT == FMT_Q6_K) {
                const uint32_t r0 = st + g * kPitch6 + w * 210u;
                if (w & 1u) q6k_block_nx<NTG, true>(r0 - 2, t, xaddr, lane, acc, release);
                else q6k_block_nx<NTG, false>(r0, t, xaddr, lane, acc, release);
            } else q80_block_nx<NTG>(st + (w >> 2) * 16 * kPitch8 + g * kPitch8 + (w & 3u) * 272u, t, xaddr, lane, acc, release);
            if (++rg.slot == rg.slots) { rg.slot = 0; rg.par ^= 1u; }
        }
        // this warp's share of the unit: rows g, g + 8 x tokens 4 tg + t (the rows' halves trade places for odd pairs of
        // tokens, which makes the stores conflict free)
        bar_wait_or_die(smem + kRedEmpty + grp8 * 8, red_par ^ 1u, a.status, dead);
        const uint32_t pp = smem + kBarBytes + (grp8 * a.red_group + w * (NTG * 64)) * 4;
#pragma unroll
        for (int tg = 0; tg < NTG; ++tg) {
            const uint32_t o = (4 * tg + t) * 16u, x = (t & 2u) << 2;
            sts32(pp + (o + (g ^ x)) * 4, acc[0][tg]);
            sts32(pp + (o + ((g + 8) ^ x)) * 4, acc[1][tg]);
        }
        __syncwarp();
        if (lane == 0) bar_arrive(smem + kRedFull + grp8 * 8);
        red_par ^= 1u;
    }
}

// FM: the formats an instance carries (bit 0 Q4_K, 1 Q6_K, 2 Q8_0): with all three in one kernel, what is live across the
// choice of the body does not fit in the registers beside the largest of them (bytes spilled: 56 with T 2 and 96 with T 4, against 0
// to 20 and 24 to 76). T: the most token groups a piece can have, 2 or 4, for the same reason (Q4_K: 8 bytes against 56).
template <int FM, int T>
__global__ void __launch_bounds__(kThreads, 1) matmul_nx_kernel(const __grid_constant__ NxArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t smem = smem_u32(smem_raw);
    // Launched as a programmatic dependent. With a table that the kernels in front write, it decides what is read at all
    // and everything waits for them; otherwise the producers start streaming the weights (constants) at once and only
    // the finalizers, which fetch the converted activations and touch y, wait.
    griddep_launch_dependents();
    if (a.table && !a.table_ready) griddep_wait();
    if (warp == 2) {   // (the second warp lists the pieces)
        if (lane < 2 * kMaxSlots) { mbar_init(bar_at(smem + kFull + 8 * lane), 1); mbar_init(bar_at(smem + kEmpty + 8 * lane), kCW); }
        fence_barrier_init();
    }
    if (tid == 0) {
        for (uint32_t i = 0; i < 2; ++i) { mbar_init(bar_at(smem + kRedFull + 8 * i), kCW); mbar_init(bar_at(smem + kRedEmpty + 8 * i), 1); }
        mbar_init(bar_at(smem + kXFull), 1);
        mbar_init(bar_at(smem + kXEmpty), kConsumers);
        fence_barrier_init();
    }
    if (warp == 3 && lane < 3 && a.t[lane].units) asm volatile("prefetch.tensormap [%0];" ::"l"(&a.map[lane]) : "memory");
    if (tid == 32) nx_list_pieces(a, smem_raw);
    __syncthreads();
    const uint32_t n_pieces = lds32(smem + kPieces), slots = lds32(smem + kPieces + 4), ring = smem + lds32(smem + kPieces + 8);
    // 640 threads start with 96 registers each: the last warpgroup (producers, finalizers) gives up 32 of them, the four
    // of the consumers take 8 more (128 x 64 + 512 x 104 = 640 x 96)
    if (warp >= kConsumers) asm volatile("setmaxnreg.dec.sync.aligned.u32 64;");
    else asm volatile("setmaxnreg.inc.sync.aligned.u32 104;");

    if (warp >= kConsumers + 2) {
        // ---- finalizers: group `grp8`'s units; the first one also brings the activation of a piece ----
        const uint32_t grp8 = warp - (kConsumers + 2);
        uint32_t red_par = 0, x_par = 1;
        griddep_wait();   // the converted activations and y come from the kernels before
#pragma unroll 1
        for (uint32_t pi = 0; pi < n_pieces; ++pi) {
            const NxPiece pc = nx_piece(smem, pi);
            const NxJob &jb = a.job[pc.job];
            const uint32_t grp = pc.grp, n_valid = pc.n_valid, tg0 = pc.tg0;
            const NxT &t = a.t[jb.tensor];
            const uint32_t ntg = (n_valid + 3) / 4, xb = xq_bytes(t.fmt), blk_bytes = ntg * xb;
            const uint8_t *img = a.xq + t.xoff + (size_t)tg0 * a.nblk * xb;
            if (grp8 == 0 && !pc.same) {   // one bulk copy per block, after the consumers left the activation before
                const uint32_t b0 = jb.seg0 * 8u, nb = min(a.nblk - b0, jb.nseg * 8u);
                if (!bar_wait(smem + kXEmpty, x_par, a.status)) return;
                fence_proxy_async_smem();
                if (lane == 0) mbar_arrive_expect_tx(bar_at(smem + kXFull), nb * blk_bytes);
                __syncwarp();
                for (uint32_t b = lane; b < nb; b += 32)
                    bulk_g2s_addr(smem + a.x_off + b * blk_bytes, img + (size_t)(b0 + b) * blk_bytes, blk_bytes, bar_at(smem + kXFull));
            }
            if (!pc.same) x_par ^= 1u;
            float inv = 1.f;   // lane p: 1 / rms of token p
            if (a.rms) {
                float ss = 0.f;
                if (lane < 4 * ntg) {
                    const uint8_t *src = img + (lane >> 2) * xb + (xb - 16) + (lane & 3u) * 4u;
#pragma unroll 8
                    for (uint32_t b = 0; b < a.nblk; ++b) ss += __ldcg(reinterpret_cast<const float *>(src + (size_t)b * blk_bytes));
                }
                inv = 1.0f / sqrtf(ss / (float)(a.nblk * 256u) + a.eps);
            }
            const float *mine = reinterpret_cast<const float *>(smem_raw + kBarBytes) + (size_t)grp8 * a.red_group;
            const bool vec = ((t.rows | t.ystride) & 3u) == 0 && ((((uintptr_t)t.y) & 15u) == 0) && (t.part_stride & 3u) == 0;
            for (uint32_t u = pc.u0 + (pc.par ^ grp8); u < pc.u1; u += 2) {
                if (!bar_wait(smem + kRedFull + grp8 * 8, red_par, a.status)) return;
                red_par ^= 1u;
                float4 v[2];
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t o = lane + 32 * i;   // outputs 4 o ..: token o / 4, rows 4 (o & 3) ..
                    v[i] = make_float4(0.f, 0.f, 0.f, 0.f);
                    if (o < 16 * ntg) {
                        const float *src = mine + 16 * (o >> 2) + ((4 * (o & 3u)) ^ (((o >> 2) & 2u) << 2));
#pragma unroll
                        for (uint32_t w = 0; w < kCW; ++w) {
                            const float4 p = *reinterpret_cast<const float4 *>(src + w * (ntg * 64));
                            v[i].x += p.x; v[i].y += p.y; v[i].z += p.z; v[i].w += p.w;
                        }
                    }
                }
                __syncwarp();
                if (lane == 0) bar_arrive(smem + kRedEmpty + grp8 * 8);
#pragma unroll
                for (int i = 0; i < 2; ++i) {
                    const uint32_t o = lane + 32 * i, tok = o >> 2, row = 16 * u + 4 * (o & 3u);
                    const float s = __shfl_sync(0xffffffffu, inv, tok & 31u);
                    if (tok >= n_valid || row >= t.rows) continue;
                    if (a.rms) { v[i].x *= s; v[i].y *= s; v[i].z *= s; v[i].w *= s; }
                    const size_t orow = a.out_idx ? a.out_idx[(size_t)grp * a.list_stride + a.col_off + tok] : pc.row0 + tok;
                    float *dst = t.y + jb.part * t.part_stride + orow * t.ystride + row;
                    if (vec) {
                        if (a.accumulate) {
                            const float4 y = *reinterpret_cast<const float4 *>(dst);
                            v[i].x += y.x; v[i].y += y.y; v[i].z += y.z; v[i].w += y.w;
                        }
                        *reinterpret_cast<float4 *>(dst) = v[i];
                    } else {
                        const float q[4] = {v[i].x, v[i].y, v[i].z, v[i].w};
#pragma unroll
                        for (int r = 0; r < 4; ++r)
                            if (row + r < t.rows) dst[r] = a.accumulate ? dst[r] + q[r] : q[r];
                    }
                }
            }
        }
        return;
    }

    if (warp >= kConsumers) {
        // ---- producers: the stages of group `grp8` ----
        const uint32_t grp8 = warp - kConsumers;
        uint32_t slot = 0, par = 1;   // a fresh barrier passes a wait on parity 1
#pragma unroll 1
        for (uint32_t pi = 0; pi < n_pieces; ++pi) {
            const NxPiece pc = nx_piece(smem, pi);
            const NxJob &jb = a.job[pc.job];
            const NxT &t = a.t[jb.tensor];
            const CUtensorMap *map = &a.map[jb.tensor];
            const uint32_t segb = seg_bytes(t.fmt);
            for (uint32_t u = pc.u0 + (pc.par ^ grp8); u < pc.u1; u += 2)
                for (uint32_t seg = 0; seg < jb.nseg; ++seg) {
                    const uint32_t off = (jb.seg0 + seg) * segb, row0 = pc.grp * t.rows + 16 * u;
                    const uint32_t bar = smem + (grp8 * kMaxSlots + slot) * 8;
                    if (!bar_wait(bar + kEmpty, par, a.status)) return;
                    fence_proxy_async_smem();
                    if (lane == 0) {
                        // 16 rows x the segment; rows past the end of the tensor and blocks past the end of a row arrive
                        // as zeros (or as another expert's rows, whose results are dropped) and count as bytes all the same
                        const uint32_t dst = ring + (grp8 * slots + slot) * a.slot_bytes;
                        uint64_t *full = bar_at(bar + kFull);
                        if (t.fmt == FMT_Q8_0) {
                            mbar_arrive_expect_tx(full, 32 * kPitch8);
                            tma_box2(dst, map, off / 8, row0, full);
                            tma_box2(dst + 16 * kPitch8, map, (off + segb / 2) / 8, row0, full);
                        } else {
                            mbar_arrive_expect_tx(full, 16 * segb);
                            if (t.swz) tma_box3(dst, map, off / 128, row0, full);
                            else tma_box2(dst, map, off / 8, row0, full);
                        }
                    }
                    if (++slot == slots) { slot = 0; par ^= 1u; }
                }
        }
        return;
    }

    // ---- consumers ----
    const uint32_t grp8 = warp / kCW, w = warp % kCW;
    NxRing rg{0, 0, slots, ring + grp8 * slots * a.slot_bytes};
    uint32_t red_par = 0, x_par = 0;
    bool dead = false;
#pragma unroll 1
    for (uint32_t pi = 0; pi < n_pieces; ++pi) {
        const NxPiece pc = nx_piece(smem, pi);
        const NxJob &jb = a.job[pc.job];
        const uint32_t u0 = pc.u0 + (pc.par ^ grp8), u1 = pc.u1;   // this group's units: every other one
        if (!pc.same) {
            if (pi) {   // done with the activation before
                __syncwarp();
                if (lane == 0) bar_arrive(smem + kXEmpty);
            }
            bar_wait_or_die(smem + kXFull, x_par, a.status, dead);
            x_par ^= 1u;
        }
        const int fmt = a.t[jb.tensor].fmt;
        const uint32_t ntg = (pc.n_valid + 3) / 4;
#define FLB_CONSUME(F, N) consume<F, N>(a, smem, jb, u0, u1, grp8, w, lane, rg, red_par, dead)
#define FLB_CONSUME_F(F)                                                                                             \
    (ntg == 1 ? FLB_CONSUME(F, 1) : T == 2 || ntg == 2 ? FLB_CONSUME(F, 2) : ntg == 3 ? FLB_CONSUME(F, 3) : FLB_CONSUME(F, 4))
        if ((FM & 1) && (FM == 1 || fmt == FMT_Q4_K)) FLB_CONSUME_F(FMT_Q4_K);
        else if ((FM & 2) && (FM == 2 || fmt == FMT_Q6_K)) FLB_CONSUME_F(FMT_Q6_K);
        else if (FM & 4) FLB_CONSUME_F(FMT_Q8_0);
#undef FLB_CONSUME_F
#undef FLB_CONSUME
    }
}

// How a launch over tensors of these formats is cut along the columns, and its shared memory. `split`: the caller adds the
// planes of the parts on the fly, so the columns are cut to one segment per part, which halves (4096 columns) the activation
// that every CTA has to load before it starts, leaves room for more stages, and doubles the number of items that are shared
// out; otherwise all columns are one part where they fit with one stage per group, or as many segments as leave two.
struct NxPlan { uint32_t parts, segs, slot_bytes, x_off, x_blk_tg; };
bool nx_plan(const int *fmts, int n, uint32_t cols, uint32_t ntg, bool split, NxPlan &p) {
    uint32_t xb = 0, slot = 0;
    for (int i = 0; i < n; ++i) { xb = std::max(xb, xq_bytes(fmts[i])); slot = std::max(slot, slot_of(fmts[i])); }
    const uint32_t nblk = cols / 256, nseg = (nblk + 7) / 8;
    p.x_off = kBarBytes + 2 * kCW * ntg * 64 * 4;
    auto fit = [&](uint32_t segs) {   // stages per group beside the activation of `segs` segments
        p.x_blk_tg = std::min(nblk, segs * 8) * xb;
        const uint32_t off = nx_ring_off(p.x_off, p.x_blk_tg, ntg);
        return off + 2 * slot <= kSmemLimit ? (kSmemLimit - off) / (2 * slot) : 0u;
    };
    uint32_t segs = split ? 1 : nseg;
    if (!split && fit(segs) < 1) {
        segs = 1;
        while (segs + 1 < nseg && fit(segs + 1) >= 2) ++segs;
        const uint32_t parts = (nseg + segs - 1) / segs;
        segs = (nseg + parts - 1) / parts;
    }
    if (fit(segs) < 1) return false;
    p.segs = segs;
    p.parts = (nseg + segs - 1) / segs;
    p.slot_bytes = slot;
    return true;
}

bool nx_tensor_ok(const NxTensor &t, uint32_t cols) {
    if ((t.fmt != FMT_Q4_K && t.fmt != FMT_Q6_K && t.fmt != FMT_Q8_0) || t.rows == 0) return false;
    const uint64_t rb = row_bytes(t.fmt, cols), pitch = t.pitch ? t.pitch : rb;
    return (pitch & 15u) == 0 && pitch >= rb && (((uintptr_t)t.w) & 15u) == 0;
}

size_t nx_image_bytes(int fmt, uint32_t cols, uint32_t tgs) { return (size_t)(cols / 256) * tgs * xq_bytes(fmt); }

// The images of a call lie one behind the other: Q4_K, Q6_K, Q8_0 (those wanted). Returns the offset of `fmt`'s.
uint32_t nx_image_off(int fmt, bool q4, bool q6, uint32_t cols, uint32_t tgs) {
    size_t o = 0;
    if (fmt != FMT_Q4_K && q4) o += nx_image_bytes(FMT_Q4_K, cols, tgs);
    if (fmt == FMT_Q8_0 && q6) o += nx_image_bytes(FMT_Q6_K, cols, tgs);
    return (uint32_t)o;
}

void (*const kNxKernels[2][5])(const NxArgs) = {
    {matmul_nx_kernel<1, 2>, matmul_nx_kernel<2, 2>, matmul_nx_kernel<3, 2>, matmul_nx_kernel<4, 2>, matmul_nx_kernel<7, 2>},
    {matmul_nx_kernel<1, 4>, matmul_nx_kernel<2, 4>, matmul_nx_kernel<3, 4>, matmul_nx_kernel<4, 4>, matmul_nx_kernel<7, 4>}};

} // namespace

cudaError_t matmul_tc_nx_init(void) {
    if (const cudaError_t e = matmul_tm_init()) return e;
    for (const auto &row : kNxKernels)
        for (auto k : row) {
            const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemLimit);
            if (e != cudaSuccess) return e;
        }
    return cudaSuccess;
}

// Bytes of device scratch the converted activations of `tgs` groups of four columns need, one image per layout.
size_t matmul_tc_nx_scratch_bytes(uint32_t cols, uint32_t tgs, int layouts) {
    return (size_t)(cols / 256) * tgs * (kXq4 + (layouts > 1 ? kXq6 : 0) + (layouts > 2 ? kXq6 : 0));
}

uint32_t matmul_tc_nx_parts(const NxTensor *t, int n, uint32_t cols, uint32_t P, bool split, int tm_sms) {
    static const bool off = getenv("FLB_TC_NX") && getenv("FLB_TC_NX")[0] == '0';
    if (off || n < 1 || n > 3 || cols % 256 != 0 || cols < 256 || cols > kNxMaxCols || P == 0 || P > kNxMaxTokens) return 0;
    int fmts[3];
    for (int i = 0; i < n; ++i) {
        if (!nx_tensor_ok(t[i], cols)) return 0;
        fmts[i] = t[i].fmt;
    }
    if (split && tm_sms && matmul_tm_takes(t, n, cols, P, tm_sms)) return matmul_tm_parts(t, n, cols, true, tm_sms);
    if (!split && tm_sms && matmul_tm_takes_whole(t, n, cols, P, tm_sms)) return 1;
    NxPlan p;
    return nx_plan(fmts, n, cols, (P + 3) / 4, split, p) ? p.parts : 0;
}

cudaError_t launch_nx_convert(const NxIn &in, const NxTensor *t, int n, uint32_t cols, uint32_t P, uint8_t *xq, uint32_t tgs_cap,
                              cudaStream_t stream, bool pdl) {
    if (cols % 256 != 0 || P == 0 || P > kNxMaxTokens || (in.xstride & 3u) || (in.rstride & 3u) || (in.part_stride & 3u)) return cudaErrorNotSupported;
    if ((((uintptr_t)in.x) | ((uintptr_t)in.x2) | ((uintptr_t)in.resid) | ((uintptr_t)in.x_out) | ((uintptr_t)in.wnorm)) & 15u) return cudaErrorNotSupported;
    bool q4 = false, q6 = false, q8 = false;
    for (int i = 0; i < n; ++i) (t[i].fmt == FMT_Q4_K ? q4 : t[i].fmt == FMT_Q6_K ? q6 : q8) = true;
    ConvArgs c{};
    c.x = in.x; c.x2 = in.x2; c.part_stride = in.part_stride; c.resid = in.resid; c.x_out = in.x_out; c.wnorm = in.wnorm;
    c.xstride = in.xstride; c.rstride = in.rstride; c.n_parts = in.n_parts ? in.n_parts : 1; c.P = P; c.nblk = cols / 256;
    c.tm = in.tm; c.dep_first = in.dep_first;
    if (in.tm && (q8 || q4 == q6 || in.table)) return cudaErrorNotSupported;
    if (in.table && (in.n_tgs == 0 || in.n_tgs > 16000)) return cudaErrorNotSupported;
    if (q4) c.img4 = xq;
    if (q6) c.img6 = xq + nx_image_off(FMT_Q6_K, q4, q6, cols, tgs_cap);
    if (q8) c.img8 = xq + nx_image_off(FMT_Q8_0, q4, q6, cols, tgs_cap);
    c.att = in.att; c.n_splits = in.n_splits;
    c.table = in.table; c.col_idx = in.col_idx; c.list_stride = in.list_stride; c.col_off = in.col_off; c.n_groups = in.n_groups;
    // Grouped, up to eight blocks an SM: each reserves an eighth of the SM's shared memory, so that they spread. They come while the matmul in
    // front leaves, and without that gather on the first SMs it frees (16 rather than 6 of them for 128 blocks; gate | up's end to the
    // conversion's, 2048 x 2048, 4 experts, 4 tokens: 4.6 -> 3.2 us; 2048 x 4096, 4 experts, 8 tokens, whole block 51.2 -> 49.2).
    // More blocks than that take what room there is (4096 x 14336, 16 tokens: 275 us, 280 with eight an SM).
    const uint32_t blocks = cols / 256 * 4 * in.n_tgs;
    const size_t reserve = in.table && blocks <= 8u * in.sms ? 24 * 1024 : 0;
    return launch_kernel(in.table ? act_convert_nx_kernel<16, true, false>
                         : in.att && in.n_splits > 16 ? (in.tm ? act_convert_nx_kernel<40, false, true> : act_convert_nx_kernel<40, false, false>)
                         : in.tm ? act_convert_nx_kernel<16, false, true> : act_convert_nx_kernel<16, false, false>, dim3(cols / 256, in.table ? 4 * in.n_tgs : (P + 3) / 4 * 4), dim3(64),
                         reserve, stream, pdl, c);
}

cudaError_t launch_nx_matmul(const NxIn &in, const NxTensor *t, int n, uint32_t cols, uint32_t P, int accumulate, const uint8_t *xq,
                             uint32_t tgs_cap, uint32_t *status, int sms, cudaStream_t stream, bool pdl, bool split) {
    if (matmul_tc_nx_parts(t, n, cols, P, split) == 0) return cudaErrorNotSupported;
    static_assert(sizeof(NxArgs) <= 4000, "kernel arguments");
    NxArgs k;
    memset(&k, 0, sizeof(k));
    int fmts[3];
    bool q4 = false, q6 = false, q8 = false;
    for (int i = 0; i < n; ++i) {
        fmts[i] = t[i].fmt;
        (t[i].fmt == FMT_Q4_K ? q4 : t[i].fmt == FMT_Q6_K ? q6 : q8) = true;
    }
    const auto kernel = kNxKernels[P > 8 ? 1 : 0][q8 ? (q4 || q6 ? 4 : 3) : (q4 ? 1 : 0) + (q6 ? 2 : 0) - 1];
    NxPlan p;
    if (!nx_plan(fmts, n, cols, (P + 3) / 4, split, p) || p.parts * n > (uint32_t)kMaxJobs) return cudaErrorNotSupported;
    const uint32_t nblk = cols / 256, nseg = (nblk + 7) / 8;
    for (int i = 0; i < n; ++i) {
        NxT &d = k.t[i];
        const uint32_t pitch = t[i].pitch ? t[i].pitch : (uint32_t)row_bytes(t[i].fmt, cols);
        const uint64_t all_rows = (uint64_t)t[i].rows * (in.table ? in.n_experts : 1);
        d.y = t[i].y; d.part_stride = p.parts > 1 ? t[i].part_stride : 0; d.rows = t[i].rows; d.ystride = t[i].ystride; d.fmt = t[i].fmt;
        d.units = (t[i].rows + 15) / 16;
        d.xoff = nx_image_off(t[i].fmt, q4, q6, cols, tgs_cap);
        d.swz = (t[i].fmt == FMT_Q4_K && pitch % 128 == 0) ? 1 : 0;
        const cudaError_t e = d.swz ? tensor_map_lines_swz(&k.map[i], t[i].w, all_rows, pitch, kSeg4 / 128, 16)
                                    : tensor_map_2d(&k.map[i], 8, t[i].w, pitch / 8, all_rows, pitch,
                                                    (t[i].fmt == FMT_Q8_0 ? kPitch8 : seg_bytes(t[i].fmt)) / 8, 16, false);
        if (e != cudaSuccess) return e;
    }
    uint64_t line = 0, items = 0;
    for (uint32_t s = 0; s < p.parts; ++s)   // the tensors of a part side by side: those of one format share its activation
        for (int i = 0; i < n; ++i) {
            NxJob &j = k.job[k.n_jobs++];
            j.tensor = (uint16_t)i; j.part = (uint16_t)s; j.seg0 = (uint16_t)(s * p.segs); j.nseg = (uint16_t)std::min(p.segs, nseg - s * p.segs);
            j.base = (uint32_t)line; j.cost = (t[i].fmt == FMT_Q4_K ? 2u : t[i].fmt == FMT_Q6_K ? 3u : 4u) * j.nseg;   // as the segments' bytes, roughly
            line += (uint64_t)k.t[i].units * j.cost;
            items += k.t[i].units;
        }
    if (line * (in.table ? in.n_groups : 1) >= (1ull << 31)) return cudaErrorNotSupported;
    k.group_cost = (uint32_t)line; k.nblk = nblk; k.P = P; k.xq = xq; k.accumulate = accumulate;
    k.rms = in.wnorm ? 1 : 0; k.eps = in.eps;
    k.red_group = kCW * ((P + 3) / 4) * 64;
    k.slot_bytes = p.slot_bytes; k.x_off = p.x_off; k.x_blk_tg = p.x_blk_tg;
    k.table = in.table; k.out_idx = in.out_idx; k.list_stride = in.list_stride; k.col_off = in.col_off; k.table_ready = in.table_ready;
    k.status = status;
    const uint32_t grid = (uint32_t)std::min<uint64_t>(items * (in.table ? in.n_groups : 1), (uint64_t)sms);
    if ((uint64_t)k.n_jobs * (in.table ? in.n_groups : 1) / grid + 2 > kMaxPieces) return cudaErrorNotSupported;
    return launch_kernel(kernel, dim3(grid), dim3(kThreads), kSmemLimit, stream, pdl, k);
}

cudaError_t launch_reduce_parts(const float *part, size_t part_stride, uint32_t n_parts, float *y, uint32_t rows, uint32_t ystride,
                                uint32_t P, int accumulate, cudaStream_t stream, bool pdl) {
    return launch_kernel(reduce_parts_kernel, dim3((rows + 255) / 256, P), dim3(256), 0, stream, pdl, part, part_stride, n_parts, y, rows,
                         ystride, accumulate);
}

} // namespace flb
