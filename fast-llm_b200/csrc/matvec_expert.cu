// The selected experts of one token (STREAM_DOT_IDX, src/runtime/runtime_internal.h:149-152): every slot's gate | up rows with the
// SwiGLU product in one launch, every slot's down rows in another, the experts' ids read on the device.
//
// HBM-bound: the rows of the slots' experts stream through shared memory once, as tiled TMA boxes of 16 rows x 2048 columns, the
// products run on mma.sync.m16n8k32 as in matvec_tc.cu (lane (g, t) holds rows g and g + 8; lane column t accumulates its own
// sub-blocks). The results are bit for bit those of the dp4a streaming kernel (matvec.cu), one launch per slot, which this
// replaces where it takes the shape: a model amplifies a difference of 1e-6 in an expert's output to 3e-5 of its logits, since
// the next block's rounding of the activation is discontinuous. (But for gate | up of more than 6144 columns, whose sum of squares lies on
// another number of warps: 1 / rms differs in its last bits, the logits by 2e-6.) Hence
//   * the activation is that kernel's: per 256-column block X = rint(x / s), s = amax / 1040000, sums of X exact in 32 bits. X
//     is cut into three balanced 8-bit digits (there: 7-bit ones for dp4a), two in the first instruction of a pair and one in the
//     second; the digit sums are put together in 32-bit integers, the same numbers as there;
//   * a warp adds the segments of a row in order, so a unit (16 rows; SwiGLU: 8 gate + 8 up) belongs to ONE of the two groups of
//     8 consumer warps, and its 32 partial sums a row (8 super-blocks x 4 lane columns) are added in that kernel's order.
// Down: a CTA serves one slot (its activation alone is in shared memory), slot k the CTAs k, k + K, ...
// Measured (Mixtral shape, 2 of 8 experts, inside the step, from the end of the launch before to its own): gate | up 44 us in
// two launches -> 24.5 in one (5.4 TB/s, the wait for the ids included), down 31 -> 15.5 (4.3 TB/s: 3.46 units a CTA are 4 rounds).
#include "common.cuh"
#include "kernels.h"
#include "tc_ops.cuh"

#include <algorithm>
#include <cstring>

namespace flb {

namespace {

constexpr int kCW = 8;                                    // consumer warps of a group, one per super-block of a segment
constexpr uint32_t kConsumers = 2 * kCW, kProducer = kConsumers, kFinal = kConsumers + 2, kThreads = (kConsumers + 4) * 32;
constexpr uint32_t kPrologueThreads = kThreads - 64;      // every warp but the producers
constexpr uint32_t kHalfWarps = 2 * (kConsumers + 2);     // of the prologue
constexpr uint32_t kSeg4 = 8 * 144, kSeg6 = 8 * 210;      // row pitch of a stage (see matvec_tc.cu)
constexpr uint32_t kSlot4 = 18 * 1024, kSlot6 = 27 * 1024;
static_assert(16 * kSeg4 <= kSlot4 && 16 * kSeg6 <= kSlot6, "slots");
constexpr uint32_t kMaxStages = 8;                        // per group
constexpr uint32_t kSmemMax = 226 * 1024;
constexpr float kFixMax = 1040000.0f;

struct ExpArgs {
    CUtensorMap map[2];          // gate and up, or down alone: the rows of all experts
    const float *x, *wnorm;      // slot k's activation: x + k * x_stride
    float *y;                    // slot k's results: y + k * rows
    const uint32_t *id;          // slot k's expert
    float eps;
    uint32_t x_stride, cols, rows, units, n_slots, stages, ring_off;   // rows, units: of one expert; stages: per group
    int swz, x_ready;
    uint32_t *status;
};

// Shared memory: barriers, sums of squares, the rows' partial sums [group][2][16 rows][8 warps][4 lane columns], the activation, the rings.
constexpr uint32_t kFullOff = 0, kEmptyOff = kFullOff + 2 * kMaxStages * 8, kRedFullOff = kEmptyOff + 2 * kMaxStages * 8,
                   kRedEmptyOff = kRedFullOff + 32, kSsqOff = kRedEmptyOff + 32, kZeroOff = kSsqOff + 96, kRedOff = kZeroOff + 32;
static_assert(kRedOff % 16 == 0 && kSsqOff + 4 * (kConsumers + 2) <= kZeroOff, "shared memory");
constexpr uint32_t kRedBytes = 16 * 32 * 4, kXOff = kRedOff + 4 * kRedBytes;
// the activation of nblk blocks: scale (f32), sums of its columns (Q4_K: 8 sub-blocks; Q6_K: 16 groups), digits (1024 bytes)
template <int F> __host__ __device__ constexpr uint32_t x_bytes(uint32_t nblk) { return ((nblk * 4 + 15) & ~15u) + nblk * (F == FMT_Q4_K ? 32 : 64) + nblk * 1024; }

__device__ __forceinline__ uint64_t *bar_at(uint8_t *base, uint32_t off) { return reinterpret_cast<uint64_t *>(base + off); }

// (digits of X as bytes) . (quants) of a lane column, from the sums over the digit planes
__device__ __forceinline__ int whole(int hi, int mid, int lo) { return hi * 65536 + mid * 256 + lo; }

// Q4_K: rows g (r0) and g + 8 of one super-block, chunk t: what the dp4a kernel's q4k_quarter gives. The loads first.
__device__ __forceinline__ void q4k_block_x21(uint32_t r0, uint32_t oh, uint32_t oa, uint32_t ob, uint32_t t, uint32_t xaddr,
                                              uint32_t xstride, float2 sx, float &out0, float &out1) {
    const uint32_t r1 = r0 + 8 * kSeg4;
    const uint4 wa0 = lds128(r0 + oa), wa1 = lds128(r1 + oa);
    uint4 bx[8];   // slot 2 m + h: (b0, b1) of the upper two digits and of the lowest for word pair m, nibble kind h
#pragma unroll
    for (int j = 0; j < 4; ++j) bx[j] = lds128(xaddr + j * xstride);
    const uint4 wb0 = lds128(r0 + ob), wb1 = lds128(r1 + ob);
#pragma unroll
    for (int j = 4; j < 8; ++j) bx[j] = lds128(xaddr + j * xstride);
    const uint4 h0 = lds128(r0 + oh), h1 = lds128(r1 + oh);
    int cL[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}}, cH[2][4] = {{0, 0, 0, 0}, {0, 0, 0, 0}};
    const uint32_t ML = 0x0F0F0F0Fu, MH = 0xF0F0F0F0u;
#pragma unroll
    for (int m = 0; m < 4; ++m) {
        const uint32_t A0 = m < 2 ? word_of(wa0, 2 * m) : word_of(wb0, 2 * m - 4), B0 = m < 2 ? word_of(wa0, 2 * m + 1) : word_of(wb0, 2 * m - 3);
        const uint32_t A1 = m < 2 ? word_of(wa1, 2 * m) : word_of(wb1, 2 * m - 4), B1 = m < 2 ? word_of(wa1, 2 * m + 1) : word_of(wb1, 2 * m - 3);
        const uint32_t l0 = A0 & ML, l1 = A1 & ML, l2 = B0 & ML, l3 = B1 & ML;
        const uint32_t g0 = A0 & MH, g1 = A1 & MH, g2 = B0 & MH, g3 = B1 & MH;   // 16 times the quants
        imma16832(cL[0], l0, l1, l2, l3, bx[2 * m].x, bx[2 * m].y);
        imma16832(cH[0], g0, g1, g2, g3, bx[2 * m + 1].x, bx[2 * m + 1].y);
        imma16832(cL[1], l0, l1, l2, l3, bx[2 * m].z, bx[2 * m].w);
        imma16832(cH[1], g0, g1, g2, g3, bx[2 * m + 1].z, bx[2 * m + 1].w);
    }
    // 6-bit scales / mins of sub-blocks 2t, 2t+1 (fl_q4k_scale_min, src/runtime/quants.h:121-129), as in matvec_tc.cu
    const uint32_t sh = 16u * (t & 1u);
    const uint32_t shA = t >= 2 ? sh + 2u : sh, mA = t >= 2 ? 0x3030u : 0x3F3Fu, mE = t >= 2 ? 0x0F0Fu : 0u;
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint4 hdr = r ? h1 : h0;
        const uint32_t sc = ((hdr.y >> shA) & mA) | ((hdr.w >> sh) & mE);
        const uint32_t mn = ((hdr.z >> shA) & mA) | ((hdr.w >> (sh + 4u)) & mE);
        const float d = h2f_bits((uint16_t)(hdr.x & 0xFFFFu)), dmin = h2f_bits((uint16_t)(hdr.x >> 16));
        const float fa = (float)whole(cL[0][2 * r], cL[0][2 * r + 1], cL[1][2 * r]);
        // the high nibbles' sums are multiples of 16, and too large for 32 bits before the division
        const float fb = (float)(cH[0][2 * r] * 4096 + cH[0][2 * r + 1] * 16 + (cH[1][2 * r] >> 4));
        const float q = dot2(u8f<0>(sc), fa, u8f<1>(sc), fb), m = dot2(u8f<0>(mn), sx.x, u8f<1>(mn), sx.y);
        (r ? out1 : out0) = dot2(d, q, -dmin, m);
    }
}

// Q6_K: lane column t = 2 hf + hq, the dp4a kernel's q6k_quarter; loads and unpacking as in matvec_tc.cu (q6k_block_i8).
template <bool ODD>
__device__ __forceinline__ void q6k_block_x21(uint32_t r0, uint32_t r1, uint32_t t, uint32_t xaddr, uint32_t xstride, float4 sx4,
                                              float &out0, float &out1) {
    const uint32_t hf = t >> 1, hq = t & 1u;
    const uint32_t oa = 64 * hf + 16 * hq, oh = 128 + 32 * hf + 16 * hq;   // byte offsets in the block
    uint32_t wa[2][4], wb[2][4], wh[2][4];
#pragma unroll
    for (int s = 0; s < 4; ++s) {
        const uint32_t js = ((uint32_t)s + t) & 3u;
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const uint32_t rb = r ? r1 : r0;
            if (ODD) {
                wa[r][s] = __byte_perm(lds32(rb + oa + 4 * js), lds32(rb + oa + 4 * js + 4), 0x5432u);
                wb[r][s] = __byte_perm(lds32(rb + oa + 32 + 4 * js), lds32(rb + oa + 36 + 4 * js), 0x5432u);
                wh[r][s] = __byte_perm(lds32(rb + oh + 4 * js), lds32(rb + oh + 4 * js + 4), 0x5432u);
            } else {
                wa[r][s] = lds32(rb + oa + 4 * js);
                wb[r][s] = lds32(rb + oa + 32 + 4 * js);
                wh[r][s] = lds32(rb + oh + 4 * js);
            }
        }
    }
    uint32_t sw[2];   // the lane column's four int8 scales plus 128
    float dd[2];
#pragma unroll
    for (int r = 0; r < 2; ++r) {
        const uint32_t rb = r ? r1 : r0, ps = rb + 192 + 8 * hf;
        uint32_t lo, hi;
        if (ODD) {
            const uint32_t s0 = lds32(ps), s1 = lds32(ps + 4), s2 = lds32(ps + 8);
            lo = __byte_perm(s0, s1, 0x5432u);
            hi = __byte_perm(s1, s2, 0x5432u);
        } else {
            lo = lds32(ps);
            hi = lds32(ps + 4);
        }
        sw[r] = __byte_perm(lo, hi, hq ? 0x7531u : 0x6420u) ^ 0x80808080u;
        dd[r] = h2f_bits((uint16_t)lds16(rb + (ODD ? 2u : 0u) + 208));
    }
    const float sx[4] = {sx4.x, sx4.y, sx4.z, sx4.w};
    float v[2], sc0[2], f0[2];
#pragma unroll
    for (int gq = 0; gq < 4; ++gq) {
        uint32_t q[2][4];
#pragma unroll
        for (int r = 0; r < 2; ++r)
#pragma unroll
            for (int s = 0; s < 4; ++s) {
                const uint32_t a = wa[r][s], b = wb[r][s], h = wh[r][s];
                q[r][s] = gq == 0 ? (a & 0x0F0F0F0Fu) | ((h << 4) & 0x30303030u) : gq == 1 ? (b & 0x0F0F0F0Fu) | ((h << 2) & 0x30303030u)
                        : gq == 2 ? ((a >> 4) & 0x0F0F0F0Fu) | (h & 0x30303030u) : ((b >> 4) & 0x0F0F0F0Fu) | ((h >> 2) & 0x30303030u);
            }
        const uint4 b0 = lds128(xaddr + gq * xstride), b1 = lds128(xaddr + (4 + gq) * xstride);
        int c0[4] = {0, 0, 0, 0}, c1[4] = {0, 0, 0, 0};
        imma16832(c0, q[0][0], q[1][0], q[0][1], q[1][1], b0.x, b0.y);
        imma16832(c1, q[0][0], q[1][0], q[0][1], q[1][1], b0.z, b0.w);
        imma16832(c0, q[0][2], q[1][2], q[0][3], q[1][3], b1.x, b1.y);
        imma16832(c1, q[0][2], q[1][2], q[0][3], q[1][3], b1.z, b1.w);
#pragma unroll
        for (int r = 0; r < 2; ++r) {
            const float f = (float)whole(c0[2 * r], c0[2 * r + 1], c1[2 * r]) - 32.f * sx[gq];
            const float sc = gq == 0 ? s8f<0>(sw[r]) : gq == 1 ? s8f<1>(sw[r]) : gq == 2 ? s8f<2>(sw[r]) : s8f<3>(sw[r]);
            if (gq == 0) { sc0[r] = sc; f0[r] = f; }
            else v[r] = gq == 1 ? dot2(sc0[r], f0[r], sc, f) : fmaf(sc, f, v[r]);
        }
    }
    out0 = dd[0] * v[0];
    out1 = dd[1] * v[1];
}

// F: the format; R: 256-column blocks a half-warp of the prologue converts; GU: gate | up with RMSNorm, or down
template <int F, int R, bool GU>
__global__ void __launch_bounds__(kThreads, 1) matvec_expert_kernel(const __grid_constant__ ExpArgs a) {
    extern __shared__ __align__(1024) uint8_t smem_raw[];
    constexpr uint32_t kSeg = F == FMT_Q4_K ? kSeg4 : kSeg6, kSlot = F == FMT_Q4_K ? kSlot4 : kSlot6;
    const uint32_t tid = threadIdx.x, lane = tid & 31u, warp = tid >> 5;
    const uint32_t nblk = a.cols / 256, nseg = (nblk + 7) / 8, S = a.stages;
    // this CTA's units: gate | up those of all slots in a row, down those of one slot
    const uint32_t slot = GU ? 0u : blockIdx.x % a.n_slots, first = GU ? blockIdx.x : blockIdx.x / a.n_slots;
    const uint32_t step = GU ? gridDim.x : (gridDim.x - slot + a.n_slots - 1) / a.n_slots, total = GU ? a.units * a.n_slots : a.units;
    const uint32_t my_units = first < total ? (total - first + step - 1) / step : 0;
    float *xs = reinterpret_cast<float *>(smem_raw + kXOff);
    float *sums = reinterpret_cast<float *>(smem_raw + kXOff + ((nblk * 4 + 15) & ~15u));
    uint8_t *img = reinterpret_cast<uint8_t *>(sums) + nblk * (F == FMT_Q4_K ? 32 : 64);
    if (tid == 0) {
        for (uint32_t i = 0; i < 2 * S; ++i) {
            mbar_init(bar_at(smem_raw, kFullOff + 8 * i), 1);
            mbar_init(bar_at(smem_raw, kEmptyOff + 8 * i), kCW);
        }
        for (uint32_t i = 0; i < 4; ++i) {
            mbar_init(bar_at(smem_raw, kRedFullOff + 8 * i), kCW);
            mbar_init(bar_at(smem_raw, kRedEmptyOff + 8 * i), 1);
        }
        *reinterpret_cast<uint4 *>(smem_raw + kZeroOff) = make_uint4(0u, 0u, 0u, 0u);
        fence_barrier_init();
    }
    __syncthreads();
    const uint32_t ring = smem_u32(smem_raw) + a.ring_off;

    if (warp >= kProducer && warp < kFinal) {
        // ---- producer of group grp: its units' stages; the experts are known once the selection has completed ----
        const uint32_t grp = warp - kProducer;
        if (GU) griddep_wait();   // (down: the launch in front started after that)
        griddep_launch_dependents();
        const uint64_t pol = l2_policy_evict_first();
        uint32_t s = 0, par = 1;   // a fresh barrier passes a wait on parity 1
        if (lane == 0)
            for (uint32_t k = grp; k < my_units; k += 2) {
                const uint32_t u = first + k * step, sl = GU ? u / a.units : slot, lu = GU ? u - sl * a.units : u;
                const uint32_t row0 = __ldcg(a.id + sl) * a.rows + lu * (GU ? 8u : 16u);
                for (uint32_t seg = 0; seg < nseg; ++seg) {
                    uint64_t *full = bar_at(smem_raw, kFullOff + 8 * (grp * S + s));
                    if (!mbar_wait_bounded(bar_at(smem_raw, kEmptyOff + 8 * (grp * S + s)), par, a.status)) return;
                    fence_proxy_async_smem();
                    const uint32_t dst = ring + (grp * S + s) * kSlot;
                    mbar_arrive_expect_tx(full, 16 * kSeg);
#pragma unroll
                    for (int j = 0; j < (GU ? 2 : 1); ++j) {   // gate rows, then up rows
                        if (F == FMT_Q4_K && a.swz) tma_box3_hint(dst + 8 * j * kSeg, &a.map[j], seg * (kSeg / 128), row0, full, pol);
                        else tma_box2_hint(dst + 8 * j * kSeg, &a.map[j], seg * (kSeg / 8), row0, full, pol);
                    }
                    if (++s == S) { s = 0; par ^= 1u; }
                }
            }
        return;
    }

    // ---- prologue: the activation as digits (the dp4a kernel's numbers) ----
    {
        const uint32_t pw = warp < kProducer ? warp : warp - 2;
        const uint32_t hw = 2 * pw + (lane >> 4), hl = lane & 15u;
        float4 ra[R][4], rb[GU ? R : 1][4];
#pragma unroll
        for (int b = 0; b < R; ++b)
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                ra[b][k] = make_float4(0.f, 0.f, 0.f, 0.f);
                if (GU) rb[b][k] = make_float4(0.f, 0.f, 0.f, 0.f);
            }
        if (GU) {
#pragma unroll
            for (int b = 0; b < R; ++b) {
                const uint32_t blk = hw + b * kHalfWarps;
                if (blk < nblk)
#pragma unroll
                    for (int k = 0; k < 4; ++k) rb[b][k] = __ldg(reinterpret_cast<const float4 *>(a.wnorm + blk * 256 + hl * 16) + k);
            }
        }
        if (!a.x_ready) griddep_wait();
#pragma unroll
        for (int b = 0; b < R; ++b) {
            const uint32_t blk = hw + b * kHalfWarps;
            if (blk < nblk)
#pragma unroll
                for (int k = 0; k < 4; ++k)
                    ra[b][k] = __ldcg(reinterpret_cast<const float4 *>(a.x + (size_t)slot * a.x_stride + blk * 256 + hl * 16) + k);
        }
        if (GU) {
            float ss = 0.f;
#pragma unroll
            for (int b = 0; b < R; ++b)
#pragma unroll
                for (int k = 0; k < 4; ++k) {
                    const float4 u = ra[b][k];
                    ss += (u.x * u.x + u.y * u.y) + (u.z * u.z + u.w * u.w);
                }
            ss = warp_sum(ss);
            if (lane == 0) reinterpret_cast<float *>(smem_raw + kSsqOff)[pw] = ss;
        }
#pragma unroll
        for (int b = 0; b < R; ++b) {
            const uint32_t blk = hw + b * kHalfWarps;
            if (2 * pw + b * kHalfWarps >= nblk) break;   // warp-uniform
            float v[16];
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                v[4 * k] = ra[b][k].x; v[4 * k + 1] = ra[b][k].y; v[4 * k + 2] = ra[b][k].z; v[4 * k + 3] = ra[b][k].w;
                if (GU) { v[4 * k] *= rb[b][k].x; v[4 * k + 1] *= rb[b][k].y; v[4 * k + 2] *= rb[b][k].z; v[4 * k + 3] *= rb[b][k].w; }
            }
            float amax = 0.f;
#pragma unroll
            for (int i = 0; i < 16; ++i) amax = fmax_nan(amax, fabsf(v[i]));
#pragma unroll
            for (int o = 8; o > 0; o >>= 1) amax = fmax_nan(amax, __shfl_xor_sync(0xffffffffu, amax, o));   // over the half-warp
            const float s = amax == 0.f ? 1.0f : amax / kFixMax;   // (a NaN among the columns makes the block's sums NaN)
            const float inv_s = 1.0f / s;
            int sum = 0;
            uint32_t V[16];   // the balanced digits of X in the low three bytes
#pragma unroll
            for (int i = 0; i < 16; ++i) {
                const int X = __float2int_rn(v[i] * inv_s);
                sum += X;
                V[i] = ((uint32_t)X + 0x00808080u) ^ 0x00808080u;
            }
            const int s32 = sum + __shfl_xor_sync(0xffffffffu, sum, 1);
            uint32_t P[4][4];   // [most significant digit, middle, lowest, none][group of four elements]
#pragma unroll
            for (int k = 0; k < 4; ++k) {
                const uint32_t t0 = __byte_perm(V[4 * k], V[4 * k + 1], 0x5140u), t1 = __byte_perm(V[4 * k + 2], V[4 * k + 3], 0x5140u);
                const uint32_t t2 = __byte_perm(V[4 * k], V[4 * k + 1], 0x6262u), t3 = __byte_perm(V[4 * k + 2], V[4 * k + 3], 0x6262u);
                P[2][k] = __byte_perm(t0, t1, 0x5410u);
                P[1][k] = __byte_perm(t0, t1, 0x7632u);
                P[0][k] = __byte_perm(t2, t3, 0x5410u);
                P[3][k] = 0u;
            }
            if (blk >= nblk) continue;   // (no shuffles from here on)
            const uint32_t base = smem_u32(img) + blk * 1024u;
            if (F == FMT_Q4_K) {
                // columns 16 hl ..: chunk c, nibble kind h, elements 16 (hl & 1) .. of the sub-block = word pairs m0, m0 + 1
                const uint32_t c = hl >> 2, h = (hl >> 1) & 1u, m0 = 2 * (hl & 1u);
#pragma unroll
                for (int mm = 0; mm < 2; ++mm)
#pragma unroll
                    for (int pl = 0; pl < 4; ++pl)
                        sts64(base + h * 128u + c * 32u + (m0 + mm) * 256u + (pl & 1) * 16u + (pl >> 1) * 8u, P[pl][2 * mm], P[pl][2 * mm + 1]);
                if ((hl & 1u) == 0) sums[blk * 8 + (hl >> 1)] = (float)s32;
            } else {
                // one scale group (half hf, group gq, run hq) of lane column 2 hf + hq, as in matvec_tc.cu
                const uint32_t hf = hl >> 3, gq = (hl >> 1) & 3u, hq = hl & 1u, t = 2 * hf + hq;
#pragma unroll
                for (int q = 0; q < 2; ++q)
#pragma unroll
                    for (int pp = 0; pp < 2; ++pp) {
                        const uint32_t a0 = hq ? P[pp][2 * q + 1] : P[pp][2 * q], a1 = hq ? P[pp][(2 * q + 2) & 3] : P[pp][2 * q + 1];
                        const uint32_t a2 = hq ? P[pp + 2][2 * q + 1] : P[pp + 2][2 * q], a3 = hq ? P[pp + 2][(2 * q + 2) & 3] : P[pp + 2][2 * q + 1];
                        sts128(base + gq * 128u + t * 32u + ((uint32_t)q ^ hf) * 512u + pp * 16u, a0, a1, a2, a3);
                    }
                sums[blk * 16 + t * 4 + gq] = (float)sum;
            }
            if (hl == 0) xs[blk] = s;
        }
        prologue_barrier(kPrologueThreads);
    }

    if (warp >= kFinal) {
        // ---- finalizer of group grp: lane (row i, lane column t); rows i and i + 8 of a unit ----
        const uint32_t grp = warp - kFinal, i = lane >> 2, t = lane & 3u;
        float inv_rms = 1.f;
        if (GU) {
            const float *ssq = reinterpret_cast<const float *>(smem_raw + kSsqOff);
            float sum = 0.f;
            for (uint32_t w = 0; w < kConsumers + 2; ++w) sum += ssq[w];   // the same order in every CTA
            inv_rms = 1.0f / sqrtf(sum / (float)a.cols + a.eps);
            if (a.x_ready) griddep_wait();   // y: what reads the results of the call before has completed
        }
        uint32_t n = 0;
        for (uint32_t k = grp; k < my_units; k += 2, ++n) {
            const uint32_t u = first + k * step, sl = GU ? u / a.units : slot, lu = GU ? u - sl * a.units : u, buf = 2 * grp + (n & 1u);
            if (!mbar_wait_bounded(bar_at(smem_raw, kRedFullOff + 8 * buf), (n >> 1) & 1u, a.status)) return;
            const float *red = reinterpret_cast<const float *>(smem_raw + kRedOff + buf * kRedBytes) + lane;   // [8 warps][16 rows][4]
            float v[2];
#pragma unroll
            for (int r = 0; r < 2; ++r) {
                float p[8];
#pragma unroll
                for (int w = 0; w < 8; ++w) p[w] = red[w * 64 + r * 32];
                v[r] = ((p[0] + p[4]) + (p[2] + p[6])) + ((p[1] + p[5]) + (p[3] + p[7]));
                v[r] += __shfl_xor_sync(0xffffffffu, v[r], 2);
                v[r] += __shfl_xor_sync(0xffffffffu, v[r], 1);
            }
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_at(smem_raw, kRedEmptyOff + 8 * buf));
            float *y = a.y + (size_t)sl * a.rows;
            if (GU) {   // fl_op_silu_mul, src/runtime/decode_params.h:267-272
                const float g = v[0] * inv_rms, up = v[1] * inv_rms;
                if (t == 0) y[8 * lu + i] = (g / (1.0f + expf(-g))) * up;
            } else if (t < 2) {
                y[16 * lu + 8 * t + i] = t ? v[1] : v[0];
            }
        }
    } else {
        // ---- consumers ----
        const uint32_t grp = warp / kCW, w = warp % kCW, g = lane >> 2, t = lane & 3u;
        const bool has_b = (g >> 1) == t;   // this lane feeds column g of the B operand; the others feed zeros
        const uint32_t xaddr = has_b ? smem_u32(img) + (2 * t + (g & 1u)) * 16u : smem_u32(smem_raw + kZeroOff);
        const uint32_t xstride = has_b ? 128u : 0u, xblk = has_b ? 1024u : 0u;
        const bool swz = F == FMT_Q4_K && a.swz;
        const uint32_t oh = q4_row_off(w * 144u, g, swz), oa = q4_row_off(w * 144u + 16u + 32u * t, g, swz),
                       ob = q4_row_off(w * 144u + 32u + 32u * t, g, swz);
        uint32_t s = 0, par = 0, n = 0;
        bool dead = false;
        for (uint32_t k = grp; k < my_units; k += 2, ++n) {
            float acc0 = 0.f, acc1 = 0.f;
#pragma unroll 1
            for (uint32_t seg = 0; seg < nseg; ++seg) {
                const uint32_t blk = seg * 8 + w;
                mbar_wait_or_die(bar_at(smem_raw, kFullOff + 8 * (grp * S + s)), par, a.status, dead);
                if (blk < nblk) {
                    const uint32_t st = ring + (grp * S + s) * kSlot;
                    float o0, o1;
                    if (F == FMT_Q4_K) {
                        const float2 sx = *reinterpret_cast<const float2 *>(sums + blk * 8 + 2 * t);
                        q4k_block_x21(st + g * kSeg4, oh, oa, ob, t, xaddr + blk * xblk, xstride, sx, o0, o1);
                    } else {
                        const float4 sx = *reinterpret_cast<const float4 *>(sums + blk * 16 + 4 * t);
                        const uint32_t r0 = st + g * kSeg6 + w * 210u;
                        if (w & 1u) q6k_block_x21<true>(r0 - 2, r0 + 8 * kSeg6 - 2, t, xaddr + blk * xblk, xstride, sx, o0, o1);
                        else q6k_block_x21<false>(r0, r0 + 8 * kSeg6, t, xaddr + blk * xblk, xstride, sx, o0, o1);
                    }
                    const float sc = xs[blk];
                    acc0 = fmaf(sc, o0, acc0);
                    acc1 = fmaf(sc, o1, acc1);
                }
                __syncwarp();
                if (lane == 0) mbar_arrive(bar_at(smem_raw, kEmptyOff + 8 * (grp * S + s)));
                if (++s == S) { s = 0; par ^= 1u; }
            }
            const uint32_t buf = 2 * grp + (n & 1u);
            mbar_wait_or_die(bar_at(smem_raw, kRedEmptyOff + 8 * buf), ((n >> 1) & 1u) ^ 1u, a.status, dead);
            float *red = reinterpret_cast<float *>(smem_raw + kRedOff + buf * kRedBytes) + w * 64 + lane;
            red[0] = acc0;
            red[32] = acc1;
            __syncwarp();
            if (lane == 0) mbar_arrive(bar_at(smem_raw, kRedFullOff + 8 * buf));
        }
    }
}

template <int F, bool GU> cudaError_t launch(const ExpertArgs &e, ExpArgs &k, int sms, cudaStream_t stream) {
    constexpr uint32_t kSeg = F == FMT_Q4_K ? kSeg4 : kSeg6, kSlot = F == FMT_Q4_K ? kSlot4 : kSlot6;
    const uint32_t nblk = e.cols / 256, rb = (uint32_t)row_bytes(F, e.cols);
    k.swz = F == FMT_Q4_K && rb % 128 == 0;
    const void *w[2] = {e.w[0], e.w[1]};
    for (int j = 0; j < (GU ? 2 : 1); ++j) {
        const uint64_t rows = (uint64_t)e.rows * e.n_experts;
        const cudaError_t r = k.swz ? tensor_map_lines_swz(&k.map[j], w[j], rows, rb, kSeg / 128, GU ? 8 : 16)
                                    : tensor_map_2d(&k.map[j], 8, w[j], rb / 8, rows, rb, kSeg / 8, GU ? 8 : 16, false);
        if (r != cudaSuccess) return r;
    }
    k.ring_off = (kXOff + x_bytes<F>(nblk) + 1023u) & ~1023u;
    k.stages = std::min(kMaxStages, (kSmemMax - k.ring_off) / (2 * kSlot));
    k.units = e.rows / (GU ? 8 : 16);
    const uint32_t grid = std::min<uint32_t>(k.units * e.n_slots, (uint32_t)sms);
    if (!GU && grid < e.n_slots) return cudaErrorNotSupported;
    const size_t smem = k.ring_off + (size_t)2 * k.stages * kSlot;
    return launch_kernel(nblk <= kHalfWarps ? matvec_expert_kernel<F, 1, GU> : matvec_expert_kernel<F, 2, GU>, dim3(grid), dim3(kThreads), smem,
                         stream, e.pdl != 0, k);
}

} // namespace

cudaError_t matvec_expert_init(void) {
    const void *kernels[] = {(const void *)matvec_expert_kernel<FMT_Q4_K, 1, true>,  (const void *)matvec_expert_kernel<FMT_Q4_K, 2, true>,
                             (const void *)matvec_expert_kernel<FMT_Q4_K, 1, false>, (const void *)matvec_expert_kernel<FMT_Q4_K, 2, false>,
                             (const void *)matvec_expert_kernel<FMT_Q6_K, 1, true>,  (const void *)matvec_expert_kernel<FMT_Q6_K, 2, true>,
                             (const void *)matvec_expert_kernel<FMT_Q6_K, 1, false>, (const void *)matvec_expert_kernel<FMT_Q6_K, 2, false>};
    for (const void *k : kernels) {
        const cudaError_t e = cudaFuncSetAttribute(k, cudaFuncAttributeMaxDynamicSharedMemorySize, (int)kSmemMax);
        if (e != cudaSuccess) return e;
    }
    return cudaSuccess;
}

// Q4_K or Q6_K rows of whole 16-byte pieces, as many columns as the prologue converts and two stages per group leave room for.
bool matvec_expert_takes(int fmt, uint32_t cols, uint32_t rows, uint32_t n_slots, uint32_t n_experts) {
    if ((fmt != FMT_Q4_K && fmt != FMT_Q6_K) || cols == 0 || cols % 256 || rows == 0 || rows % 16 || row_bytes(fmt, cols) % 16) return false;
    if (cols / 256 > 2 * kHalfWarps || n_slots == 0 || (uint64_t)rows * std::max(n_slots, n_experts) >= (1ull << 31)) return false;
    const uint32_t nblk = cols / 256, x = fmt == FMT_Q4_K ? x_bytes<FMT_Q4_K>(nblk) : x_bytes<FMT_Q6_K>(nblk);
    return ((kXOff + x + 1023u) & ~1023u) + 4 * (fmt == FMT_Q4_K ? kSlot4 : kSlot6) <= kSmemMax;
}

cudaError_t launch_matvec_expert(const ExpertArgs &e, int sms, cudaStream_t stream) {
    if (!matvec_expert_takes(e.fmt, e.cols, e.rows, e.n_slots, e.n_experts) || (uint32_t)sms < e.n_slots) return cudaErrorNotSupported;
    ExpArgs k;
    memset(&k, 0, sizeof(k));
    k.x = e.x; k.wnorm = e.wnorm; k.y = e.y; k.id = e.id; k.eps = e.eps; k.x_stride = e.x_stride;
    k.cols = e.cols; k.rows = e.rows; k.n_slots = e.n_slots; k.x_ready = e.x_ready; k.status = e.status;
    const bool gu = e.w[1] != nullptr;
    if (gu != (e.wnorm != nullptr)) return cudaErrorNotSupported;
    if (e.fmt == FMT_Q4_K) return gu ? launch<FMT_Q4_K, true>(e, k, sms, stream) : launch<FMT_Q4_K, false>(e, k, sms, stream);
    return gu ? launch<FMT_Q6_K, true>(e, k, sms, stream) : launch<FMT_Q6_K, false>(e, k, sms, stream);
}

} // namespace flb
