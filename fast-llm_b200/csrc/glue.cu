// Small decode operators around the matvecs and attention. Each follows one
// canonical operator of the reference (src/runtime/decode_params.h) and keeps
// its rounding where that is cheap: separate multiplies / adds via __fmul_rn,
// __fadd_rn, __fsub_rn, IEEE division and square root.
#include "common.cuh"
#include "kernels.h"

namespace flb {

namespace {

// fl_op_rmsnorm, decode_params.h:101-106. The sum of squares is a tree
// reduction here (the reference sums sequentially); everything after it rounds
// like the reference: 1/sqrtf(ss/n + eps), then (x*s)*w.
__global__ void __launch_bounds__(1024) rmsnorm_kernel(const float *__restrict__ x, const float *__restrict__ w,
                                                       float *__restrict__ y, float eps, uint32_t n, uint32_t stride) {
    __shared__ float red[32];
    __shared__ float inv;
    x += (size_t)blockIdx.y * stride;   // one block per vector
    y += (size_t)blockIdx.y * stride;
    float ss = 0.f;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) ss = fmaf(x[i], x[i], ss);
    ss = warp_sum(ss);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = ss;
    __syncthreads();
    if (threadIdx.x == 0) {
        float t = 0.f;
        for (uint32_t k = 0; k < (blockDim.x + 31) / 32; ++k) t += red[k];
        inv = 1.0f / sqrtf(__fadd_rn(t / (float)n, eps));
    }
    __syncthreads();
    const float s = inv;
    for (uint32_t i = threadIdx.x; i < n; i += blockDim.x) y[i] = __fmul_rn(__fmul_rn(x[i], s), w[i]);
}

// fl_op_add2, decode_params.h:108-110
__global__ void add2_kernel(const float *__restrict__ a, const float *__restrict__ b, float *__restrict__ y,
                            uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) y[i] = __fadd_rn(a[i], b[i]);
}

// Expert selection of the MoE router (fl_op_router_sel, src/runtime/decode_params.h:234-265): softmax over the
// expert logits of a token, the top_k largest weights (ties go to the lower index), optionally renormalised
// over the chosen ones. One warp per token, every token of the block in one launch. What the warp does in
// parallel: the maximum, the exponentials, the divisions and each round's arg-max. What stays sequential,
// because f32 sums depend on their order and the results have to equal the reference's bit for bit: the sum of
// the exponentials (ascending expert index, one lane) and the sum of the chosen weights (selection order).
// With expert parallelism (lids != nullptr) the kernel also writes, per (token, slot), the index of the expert
// among this rank's experts [base, base + n_local) or the skip mark, and the gate or 0.
struct RouterOut { uint32_t *ids; float *gates; uint32_t *lids; float *mgates; uint32_t top_k, norm; float scale; uint32_t base, n_local; };
// One warp; w, gk: n_expert and top_k floats of shared memory. The logits may come from other blocks of the launch.
__device__ __forceinline__ void router_select(const float *l, float *w, float *gk, uint32_t lane, size_t tok, uint32_t n_expert, const RouterOut &o) {
    uint32_t *ids = o.ids, *lids = o.lids;
    float *gates = o.gates, *mgates = o.mgates;
    const uint32_t top_k = o.top_k;
    float mx = -1e30f;
    for (uint32_t i = lane; i < n_expert; i += 32) mx = fmaxf(mx, __ldcg(l + i));
    mx = warp_max(mx);
    for (uint32_t i = lane; i < n_expert; i += 32) w[i] = expf(__fsub_rn(__ldcg(l + i), mx));
    __syncwarp();
    float sum = 0.f;
    if (lane == 0)
        for (uint32_t i = 0; i < n_expert; ++i) sum = __fadd_rn(sum, w[i]);
    sum = __shfl_sync(0xffffffffu, sum, 0);
    for (uint32_t i = lane; i < n_expert; i += 32) w[i] = __fdiv_rn(w[i], sum);
    __syncwarp();
    float tsum = 0.f;
    for (uint32_t k = 0; k < top_k; ++k) {
        // the largest weight not chosen yet; a chosen entry is overwritten with -2, below the starting value -1
        float bw = -1.f;
        uint32_t best = 0;
        for (uint32_t i = lane; i < n_expert; i += 32)
            if (w[i] > bw) { bw = w[i]; best = i; }
#pragma unroll
        for (int o = 16; o > 0; o >>= 1) {
            const float ow = __shfl_xor_sync(0xffffffffu, bw, o);
            const uint32_t ob = __shfl_xor_sync(0xffffffffu, best, o);
            if (ow > bw || (ow == bw && ob < best)) { bw = ow; best = ob; }
        }
        tsum = __fadd_rn(tsum, bw);   // every lane keeps the same running sum, in selection order
        if (lane == 0) {
            ids[tok * top_k + k] = best;
            gk[k] = bw;
            if (bw >= 0.f) w[best] = -2.f;
        }
        __syncwarp();
    }
    for (uint32_t k = lane; k < top_k; k += 32) {
        float g = gk[k];
        if (o.norm) g = __fdiv_rn(g, tsum);
        g = __fmul_rn(g, o.scale);
        gates[tok * top_k + k] = g;
        if (lids) {
            const uint32_t e = ids[tok * top_k + k];
            const bool mine = e >= o.base && e - o.base < o.n_local;
            lids[tok * top_k + k] = mine ? e - o.base : kExpertSkip;
            mgates[tok * top_k + k] = mine ? g : 0.f;
        }
    }
}

constexpr int kRouterWarps = 4;
__global__ void __launch_bounds__(kRouterWarps * 32) router_sel_kernel(const float *__restrict__ logits, uint32_t n_tok, uint32_t n_expert, RouterOut o) {
    __shared__ float w_s[kRouterWarps][256], g_s[kRouterWarps][256];
    const uint32_t warp = threadIdx.x >> 5, lane = threadIdx.x & 31u;
    const uint32_t tok = blockIdx.x * kRouterWarps + warp;
    if (tok >= n_tok) return;
    router_select(logits + (size_t)tok * n_expert, w_s[warp], g_s[warp], lane, tok, n_expert, o);
}

// The table of a grouped multi-column launch (matvec_tc_nx.cu), by one warp: active experts in ascending order, their
// columns from col_off on (at most P), the groups of four columns in front of them and the columns in front of them.
__device__ __forceinline__ void nx_table_warp(const uint32_t *cnt, uint32_t n_local, uint32_t col_off, uint32_t P, uint32_t *table) {
    const uint32_t lane = threadIdx.x & 31u;
    uint32_t n_act = 0, before = 0, most = 0;   // before: groups of four, columns << 16
    for (uint32_t b = 0; b < n_local; b += 32) {
        const uint32_t e = b + lane, c = e < n_local ? cnt[e] : 0u;
        const uint32_t n = c > col_off ? min(c - col_off, P) : 0u, tg = (n + 3) / 4, own = tg | n << 16;
        uint32_t incl = own;
#pragma unroll
        for (int o = 1; o < 32; o <<= 1) {
            const uint32_t v = __shfl_up_sync(0xffffffffu, incl, o);
            if (lane >= (uint32_t)o) incl += v;
        }
        const uint32_t mask = __ballot_sync(0xffffffffu, n != 0), at = before + incl - own;
        if (n) reinterpret_cast<uint4 *>(table)[1 + n_act + __popc(mask & ((1u << lane) - 1u))] = make_uint4(e, n, at & 0xFFFFu, at >> 16);
        n_act += __popc(mask);
        most = max(most, __reduce_max_sync(0xffffffffu, tg));
        before += __shfl_sync(0xffffffffu, incl, 31);
    }
    if (lane == 0) { table[0] = n_act; table[1] = most; }
}

// One warp: a stable counting sort of the (token, slot) pairs by local expert (within an expert they stay in ascending order).
// The counts in shared memory (in device memory every expert was a round trip: 3 us for 8 of them).
__global__ void __launch_bounds__(32) group_by_expert_kernel(const uint32_t *lids, uint32_t n_pairs, uint32_t top_k, uint32_t n_local, uint32_t cap,
                                                             uint32_t *cnt, uint32_t *tok_list, uint32_t *pair_list, uint32_t *table) {
    __shared__ uint32_t n_s[256];
    const uint32_t lane = threadIdx.x;
    griddep_launch_dependents();
    griddep_wait();
    for (uint32_t e = lane; e < n_local; e += 32) n_s[e] = 0;
    __syncwarp();
    for (uint32_t b = 0; b < n_pairs; b += 32) {
        const uint32_t pair = b + lane;
        const uint32_t e = pair < n_pairs ? __ldcg(lids + pair) : 0xFFFFFFFFu;
        for (uint32_t x = 0; x < n_local; ++x) {
            const uint32_t mask = __ballot_sync(0xffffffffu, e == x);
            if (mask == 0) continue;
            const uint32_t base = n_s[x];
            if (e == x) {
                const uint32_t pos = base + __popc(mask & ((1u << lane) - 1u));
                if (pos < cap) { tok_list[(size_t)x * cap + pos] = pair / top_k; pair_list[(size_t)x * cap + pos] = pair; }
            }
            __syncwarp();
            if (lane == 0) n_s[x] = min(base + __popc(mask), cap);
            __syncwarp();
        }
    }
    for (uint32_t e = lane; e < n_local; e += 32) cnt[e] = n_s[e];
    nx_table_warp(n_s, n_local, 0, kNxMaxTokens, table);
}

// Router of a block: logits[t][e] = dot(router[e], x[t]), one block per (expert, token), and the selection by the block that is the
// last of its token. wnorm != nullptr: x is the raw hidden state and the logits are those of RMSNorm(x) * wnorm (fl_op_rmsnorm,
// src/runtime/decode_params.h:101-106, fused: every block norms the token itself). Bound by latency: the router's rows and the norm
// weights are requested before the dependency, the selection saves a launch (8 experts of 4096 columns, one token, inside a
// step: 10.1 us in two launches -> 5.4; the grouping of several tokens' pairs in here too cost more than its launch, 12.4 us).
// AFTER: nothing is read before the dependency is met.
template <bool AFTER>
__global__ void __launch_bounds__(128) router_kernel(const RouterArgs a) {
    __shared__ float red[4], w_s[256], g_s[256];
    __shared__ uint32_t last;
    constexpr int kAhead = 8;   // 16-byte pieces a thread requests up front
    const uint32_t e = blockIdx.x, t = blockIdx.y, n4 = a.n_embd / 4;
    const float4 *w = reinterpret_cast<const float4 *>(a.router + (size_t)e * a.n_embd);
    const float4 *v = reinterpret_cast<const float4 *>(a.x + (size_t)t * a.n_embd);
    const float4 *gn = reinterpret_cast<const float4 *>(a.wnorm);
    float4 wa[kAhead], ga[kAhead], xa[kAhead];
#pragma unroll
    for (int k = 0; k < kAhead; ++k) {
        const uint32_t i = threadIdx.x + 128 * k;
        wa[k] = ga[k] = xa[k] = make_float4(0.f, 0.f, 0.f, 0.f);
        if (i < n4 && !AFTER) { wa[k] = __ldg(w + i); if (gn) ga[k] = __ldg(gn + i); }
    }
    griddep_wait();
    if (AFTER)
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const uint32_t i = threadIdx.x + 128 * k;
            if (i < n4) { wa[k] = __ldcg(w + i); if (gn) ga[k] = __ldcg(gn + i); }
        }
    griddep_launch_dependents();   // what starts now may take x for complete (ExpertArgs::x_ready)
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
        if (threadIdx.x + 128 * k < n4) xa[k] = v[threadIdx.x + 128 * k];
    float inv_rms = 1.f;
    if (gn) {
        float ss = 0.f;
#pragma unroll
        for (int k = 0; k < kAhead; ++k) {
            const float4 b = xa[k];
            ss += (b.x * b.x + b.y * b.y) + (b.z * b.z + b.w * b.w);
        }
        for (uint32_t i = threadIdx.x + 128 * kAhead; i < n4; i += 128) {
            const float4 b = v[i];
            ss += (b.x * b.x + b.y * b.y) + (b.z * b.z + b.w * b.w);
        }
        ss = warp_sum(ss);
        if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = ss;
        __syncthreads();
        inv_rms = 1.0f / sqrtf(((red[0] + red[1]) + (red[2] + red[3])) / (float)a.n_embd + a.eps);
        __syncthreads();
    }
    float acc = 0.f;
    auto add = [&](const float4 &r, float4 b, const float4 &g) {
        if (gn) { b.x = b.x * inv_rms * g.x; b.y = b.y * inv_rms * g.y; b.z = b.z * inv_rms * g.z; b.w = b.w * inv_rms * g.w; }
        acc = fmaf(r.x, b.x, acc); acc = fmaf(r.y, b.y, acc); acc = fmaf(r.z, b.z, acc); acc = fmaf(r.w, b.w, acc);
    };
#pragma unroll
    for (int k = 0; k < kAhead; ++k)
        if (threadIdx.x + 128 * k < n4) add(wa[k], xa[k], ga[k]);
    for (uint32_t i = threadIdx.x + 128 * kAhead; i < n4; i += 128) add(w[i], v[i], gn ? gn[i] : make_float4(0.f, 0.f, 0.f, 0.f));
    acc = warp_sum(acc);
    if ((threadIdx.x & 31u) == 0) red[threadIdx.x >> 5] = acc;
    __syncthreads();
    if (threadIdx.x == 0) {
        a.logits[(size_t)t * a.n_expert + e] = (red[0] + red[1]) + (red[2] + red[3]);
        __threadfence();
        last = atomicAdd(a.tickets + t, 1u) == a.n_expert - 1 ? 1u : 0u;
        if (last) { __threadfence(); a.tickets[t] = 0; }   // for the next launch
    }
    __syncthreads();
    if (!last || threadIdx.x >= 32) return;
    const RouterOut o{a.ids, a.gates, a.lids, a.mgates, a.top_k, a.norm, a.scale, a.base, a.n_local};
    router_select(a.logits + (size_t)t * a.n_expert, w_s, g_s, threadIdx.x, t, a.n_expert, o);
}

// fl_op_wmerge, decode_params.h:274-295: y = add1 + add2 + scale * sum_q gate_q * part_q,
// products and sums rounded separately and in the reference's order.
__global__ void wmerge_kernel(const float *__restrict__ parts, const float *__restrict__ gates,
                              const float *__restrict__ add1, const float *__restrict__ add2, float *__restrict__ y,
                              float scale, uint32_t n_parts, uint32_t n, uint32_t n_full) {
    griddep_launch_dependents();
    griddep_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i >= n) return;
    float gsc = 1.0f;
    if (gates && n_full > n_parts) {
        float s = 0.f, sf = 0.f;
        for (uint32_t q = 0; q < n_parts; ++q) s = __fadd_rn(s, gates[q]);
        for (uint32_t q = 0; q < n_full; ++q) sf = __fadd_rn(sf, gates[q]);
        if (s > 0.f) gsc = __fdiv_rn(sf, s);
    }
    float acc = 0.f;
    for (uint32_t q = 0; q < n_parts; ++q) {
        const float g = gates ? __fmul_rn(gsc, gates[q]) : 1.0f;
        acc = __fadd_rn(acc, __fmul_rn(g, parts[(size_t)q * n + i]));
    }
    acc = __fmul_rn(acc, scale);
    if (add1) acc = __fadd_rn(acc, add1[i]);
    if (add2) acc = __fadd_rn(acc, add2[i]);
    y[i] = acc;
}

// y[t][i] = (resid[t][i] +) sum_q (gates[t][q] * parts[t][q][i]), the arithmetic of fl_op_wmerge (decode_params.h:274-295)
// with one residual term at most, for every token of a block in one launch. grid (ceil(n / 256), n_tok).
__global__ void wmerge_tokens_kernel(const float *__restrict__ parts, const float *__restrict__ gates, float *y, uint32_t n_parts,
                                     uint32_t n, uint32_t n_planes, size_t plane_stride, const float *resid,
                                     const uint32_t *__restrict__ lids) {
    griddep_launch_dependents();
    griddep_wait();
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x, t = blockIdx.y;
    if (i >= n) return;
    float acc = 0.f;
#pragma unroll 2
    for (uint32_t q = 0; q < n_parts; ++q) {
        if (lids && lids[(size_t)t * n_parts + q] == kExpertSkip) continue;   // another rank's: gate 0, and no part was made here
        const float *p = parts + ((size_t)t * n_parts + q) * n + i;
        float w[kMaxPlanes];   // all planes requested before the first is used
#pragma unroll
        for (uint32_t s = 0; s < kMaxPlanes; ++s) w[s] = s < n_planes ? p[s * plane_stride] : 0.f;
        float v = w[0];
#pragma unroll
        for (uint32_t s = 1; s < kMaxPlanes; ++s)
            if (s < n_planes) v = __fadd_rn(v, w[s]);
        acc = __fadd_rn(acc, __fmul_rn(gates[(size_t)t * n_parts + q], v));
    }
    if (resid) acc = __fadd_rn(resid[(size_t)t * n + i], acc);
    y[(size_t)t * n + i] = acc;
}

// grid (ceil(n / 1024), P, groups): see launch_scatter_rows.
__global__ void __launch_bounds__(256) scatter_rows_kernel(const float *__restrict__ x, uint32_t n_planes, size_t plane_stride,
                                                           const uint32_t *__restrict__ table, const uint32_t *__restrict__ idx,
                                                           uint32_t list_stride, uint32_t col_off, float *__restrict__ y, uint32_t n) {
    const uint32_t i = 4 * (blockIdx.x * 256 + threadIdx.x), p = blockIdx.y;
    if (i >= n || blockIdx.z >= table[0]) return;
    const uint4 e = reinterpret_cast<const uint4 *>(table)[1 + blockIdx.z];
    if (p >= e.y) return;
    const float *src = x + (size_t)(e.w + p) * n + i;
    float4 v = *reinterpret_cast<const float4 *>(src);
#pragma unroll 4
    for (uint32_t s = 1; s < n_planes; ++s) {
        const float4 w = *reinterpret_cast<const float4 *>(src + s * plane_stride);
        v.x = __fadd_rn(v.x, w.x); v.y = __fadd_rn(v.y, w.y); v.z = __fadd_rn(v.z, w.z); v.w = __fadd_rn(v.w, w.w);
    }
    *reinterpret_cast<float4 *>(y + (size_t)idx[(size_t)e.x * list_stride + col_off + p] * n + i) = v;
}

__global__ void __launch_bounds__(32) nx_table_kernel(const uint32_t *__restrict__ cnt, uint32_t n_local, uint32_t col_off, uint32_t P,
                                                      uint32_t *__restrict__ table) {
    nx_table_warp(cnt, n_local, col_off, P, table);
}

// fl_op_silu_mul, decode_params.h:267-272: (g / (1 + expf(-g))) * u
__global__ void silu_mul_kernel(const float *__restrict__ g, const float *__restrict__ u, float *__restrict__ h,
                                uint32_t n) {
    const uint32_t i = blockIdx.x * blockDim.x + threadIdx.x;
    if (i < n) {
        const float v = g[i];
        h[i] = __fmul_rn(v / __fadd_rn(1.0f, expf(-v)), u[i]);
    }
}

// fl_op_rope_ds2 (decode_params.h:124-160, plain RoPE: adjacent pairs, angle
// pos * theta_scale^i built by repeated multiplication exactly as the reference
// does, so the angle is bit-identical; cosf/sinf differ from the host libm by at
// most a few ulp) followed by the f16 KV append (fl_op_kv_append,
// decode_params.h:162-175, with the cache kept in f16, head-major).
__global__ void __launch_bounds__(128) rope_append_kernel(const RopeAppendArgs a) {
    griddep_launch_dependents();
    griddep_wait();
    const uint32_t half = a.head_dim / 2;
    const uint32_t t = blockIdx.x * blockDim.x + threadIdx.x;
    const uint32_t n_rot_heads = (a.q ? a.n_q_head : 0) + a.n_kv_head;
    const uint32_t tokn = blockIdx.y;   // token of a batch pass (0 in a single step)
    const uint32_t pos = (uint32_t)a.pos[tokn];
    auto pair = [&](const float *v, float &x0, float &x1) {   // two neighbours, the planes added in order
        x0 = v[0]; x1 = v[1];
        for (uint32_t p = 1; p < a.n_planes; ++p) { x0 += v[p * a.plane_stride]; x1 += v[p * a.plane_stride + 1]; }
    };
    if (t < n_rot_heads * half) {
        const uint32_t h = t / half, i = t % half;
        float c, s;
        if (a.table) {
            const float2 cs = a.table[(size_t)tokn * half + i];
            c = cs.x; s = cs.y;
        } else {
            float theta = (float)(int32_t)pos;
            for (uint32_t k = 0; k < i; ++k) theta = __fmul_rn(theta, a.theta_scale);
            c = cosf(theta); s = sinf(theta);
        }
        const uint32_t nq = a.q ? a.n_q_head : 0;
        if (h < nq) {
            float *v = a.q + (size_t)tokn * a.q_tok_stride + (size_t)h * a.head_dim + 2 * i;
            float x0, x1;
            pair(v, x0, x1);
            v[0] = __fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s));
            v[1] = __fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c));
        } else {
            const uint32_t hk = h - nq;
            const float *v = a.k + (size_t)tokn * a.kv_tok_stride + (size_t)hk * a.head_dim + 2 * i;
            float x0, x1;
            pair(v, x0, x1);
            __half *dst = a.kcache + (size_t)tokn * a.seq_elems + ((size_t)hk * a.kv_stride + pos) * a.head_dim + 2 * i;
            dst[0] = __float2half_rn(__fsub_rn(__fmul_rn(x0, c), __fmul_rn(x1, s)));
            dst[1] = __float2half_rn(__fadd_rn(__fmul_rn(x0, s), __fmul_rn(x1, c)));
        }
    } else if (t < (n_rot_heads + a.n_kv_head) * half) {
        const uint32_t u = t - n_rot_heads * half;
        const uint32_t hk = u / half, i = u % half;
        const float *v = a.v + (size_t)tokn * a.kv_tok_stride + (size_t)hk * a.head_dim + 2 * i;
        __half *dst = a.vcache + (size_t)tokn * a.seq_elems + ((size_t)hk * a.kv_stride + pos) * a.head_dim + 2 * i;
        float x0, x1;
        pair(v, x0, x1);
        dst[0] = __float2half_rn(x0);
        dst[1] = __float2half_rn(x1);
    }
}

__global__ void rope_table_kernel(const int32_t *pos, float theta_scale, uint32_t half, float2 *table) {
    const uint32_t i = threadIdx.x;
    if (i >= half) return;
    pos += blockIdx.x;
    table += (size_t)blockIdx.x * half;
    float theta = (float)*pos;
    for (uint32_t k = 0; k < i; ++k) theta = __fmul_rn(theta, theta_scale);
    table[i] = make_float2(cosf(theta), sinf(theta));
}

// Greedy argmax: strict '>' scan order of the reference (lowest index wins
// ties) and the runner-up value for the margin (src/model/decoder.cpp:1253-1264).
struct Top { float b; uint32_t i; float s; };

__device__ __forceinline__ Top top_merge(const Top &x, const Top &y) {
    const bool y_wins = y.b > x.b || (y.b == x.b && y.i < x.i);
    Top r;
    if (y_wins) { r.b = y.b; r.i = y.i; r.s = fmaxf(x.b, fmaxf(x.s, y.s)); }
    else { r.b = x.b; r.i = x.i; r.s = fmaxf(y.b, fmaxf(x.s, y.s)); }
    return r;
}
__device__ __forceinline__ Top top_warp(Top t) {
#pragma unroll
    for (int o = 16; o > 0; o >>= 1) {
        Top u;
        u.b = __shfl_xor_sync(0xffffffffu, t.b, o);
        u.i = __shfl_xor_sync(0xffffffffu, t.i, o);
        u.s = __shfl_xor_sync(0xffffffffu, t.s, o);
        t = top_merge(t, u);
    }
    return t;
}

__global__ void __launch_bounds__(256) argmax_kernel(const float *__restrict__ lg, uint32_t n, int32_t *out_idx,
                                                     float *out_margin, float *scratch, uint32_t *ticket, float *top3) {
    griddep_launch_dependents();
    griddep_wait();
    const uint32_t row = blockIdx.y;   // one row of logits per block row
    lg += (size_t)row * n;
    out_idx += row; out_margin += row; ticket += row;
    scratch += (size_t)row * kArgmaxScratch;
    if (top3) top3 += 4 * row;
    __shared__ Top wtop[8];
    __shared__ uint32_t last;
    Top t{-INFINITY, 0xFFFFFFFFu, -INFINITY};
    for (uint32_t i = blockIdx.x * blockDim.x + threadIdx.x; i < n; i += gridDim.x * blockDim.x) {
        const float v = lg[i];
        if (v > t.b) { t.s = t.b; t.b = v; t.i = i; }   // indices ascend within a thread
        else if (v > t.s) t.s = v;
    }
    t = top_warp(t);
    if ((threadIdx.x & 31u) == 0) wtop[threadIdx.x >> 5] = t;
    __syncthreads();
    if (threadIdx.x == 0) {
        Top r = wtop[0];
        for (int w = 1; w < 8; ++w) r = top_merge(r, wtop[w]);
        float *slot = scratch + 3 * blockIdx.x;
        slot[0] = r.b; slot[1] = __uint_as_float(r.i); slot[2] = r.s;
        __threadfence();
        last = atomicAdd(ticket, 1u) == gridDim.x - 1 ? 1u : 0u;
    }
    __syncthreads();
    if (!last) return;
    __threadfence();
    if (threadIdx.x < 32) {
        Top r{-INFINITY, 0xFFFFFFFFu, -INFINITY};
        for (uint32_t k = threadIdx.x; k < gridDim.x; k += 32) {
            Top u;
            u.b = __ldcg(scratch + 3 * k);
            u.i = __float_as_uint(__ldcg(scratch + 3 * k + 1));
            u.s = __ldcg(scratch + 3 * k + 2);
            r = top_merge(r, u);
        }
        r = top_warp(r);
        if (threadIdx.x == 0) {
            *out_idx = (int32_t)r.i;
            *out_margin = r.b - r.s;
            if (top3) { top3[0] = r.b; top3[1] = __uint_as_float(r.i); top3[2] = r.s; }   // for the cross-rank merge
            *ticket = 0;
        }
    }
}

// Bound by its launch: a few hundred kilobytes at most in earnest (16 bytes a thread and round).
__global__ void __launch_bounds__(256) fill_kernel(uint8_t *dst, uint32_t v, size_t bytes, uint32_t head) {
    griddep_launch_dependents();
    griddep_wait();
    uint4 *mid = reinterpret_cast<uint4 *>(dst + head);
    const size_t n16 = (bytes - head) / 16, tail = head + 16 * n16;
    const uint4 q = make_uint4(v, v, v, v);
    for (size_t i = blockIdx.x * (size_t)256 + threadIdx.x; i < n16; i += (size_t)gridDim.x * 256) mid[i] = q;
    if (blockIdx.x == 0 && threadIdx.x < 32) {   // the bytes in front of the first and behind the last whole 16
        if (threadIdx.x < head) dst[threadIdx.x] = (uint8_t)v;
        if (tail + threadIdx.x < bytes && threadIdx.x < 16) dst[tail + threadIdx.x] = (uint8_t)v;
    }
}

} // namespace

cudaError_t launch_fill(void *dst, int value, size_t bytes, int sms, cudaStream_t stream, bool pdl) {
    if (!dst || !bytes) return cudaErrorInvalidValue;
    const uint32_t head = (uint32_t)std::min<size_t>((16 - ((uintptr_t)dst & 15u)) & 15u, bytes);
    const uint32_t grid = (uint32_t)std::min<size_t>(bytes / 4096 + 1, (size_t)8 * sms);
    return launch_kernel(fill_kernel, dim3(grid), dim3(256), 0, stream, pdl, (uint8_t *)dst, (uint32_t)(uint8_t)value * 0x01010101u, bytes, head);
}

cudaError_t launch_rmsnorm(const float *x, const float *wnorm, float *y, float eps, uint32_t n,
                           cudaStream_t stream, uint32_t rows, uint32_t stride) {
    if (rows == 0) return cudaErrorInvalidValue;
    rmsnorm_kernel<<<dim3(1, rows), 1024, 0, stream>>>(x, wnorm, y, eps, n, stride);
    return cudaGetLastError();
}

cudaError_t launch_add2(const float *a, const float *b, float *y, uint32_t n, cudaStream_t stream) {
    add2_kernel<<<(n + 255) / 256, 256, 0, stream>>>(a, b, y, n);
    return cudaGetLastError();
}

cudaError_t launch_router_sel(const float *logits, uint32_t *ids, float *gates, uint32_t n_tok, uint32_t n_expert, uint32_t top_k,
                              uint32_t norm, float scale, cudaStream_t stream, uint32_t *lids, float *mgates, uint32_t base,
                              uint32_t n_local) {
    if (n_tok == 0 || n_expert == 0 || n_expert > 256 || top_k == 0 || top_k > n_expert) return cudaErrorInvalidValue;
    if ((lids == nullptr) != (mgates == nullptr)) return cudaErrorInvalidValue;
    router_sel_kernel<<<(n_tok + kRouterWarps - 1) / kRouterWarps, kRouterWarps * 32, 0, stream>>>(
        logits, n_tok, n_expert, RouterOut{ids, gates, lids, mgates, top_k, norm, scale, base, n_local});
    return cudaGetLastError();
}

cudaError_t launch_router(const RouterArgs &a, cudaStream_t stream) {
    if (a.n_tok == 0 || a.n_expert == 0 || a.n_expert > 256 || a.top_k == 0 || a.top_k > a.n_expert || a.n_embd % 4) return cudaErrorInvalidValue;
    return launch_kernel(a.w_after ? router_kernel<true> : router_kernel<false>, dim3(a.n_expert, a.n_tok), dim3(128), 0, stream, a.pdl != 0, a);
}

cudaError_t launch_wmerge(const float *parts, const float *gates, const float *add1, const float *add2, float *y,
                          float scale, uint32_t n_parts, uint32_t n, uint32_t n_full, cudaStream_t stream, bool pdl) {
    if (n == 0 || n_parts == 0) return cudaErrorInvalidValue;
    return launch_kernel(wmerge_kernel, dim3((n + 255) / 256), dim3(256), 0, stream, pdl, parts, gates, add1, add2, y, scale, n_parts, n, n_full);
}

cudaError_t launch_wmerge_tokens(const float *parts, const float *gates, float *y, uint32_t n_parts, uint32_t n, uint32_t n_tok,
                                 cudaStream_t stream, uint32_t n_planes, size_t plane_stride, const float *resid, const uint32_t *lids, bool pdl) {
    if (n == 0 || n_parts == 0 || n_tok == 0) return cudaErrorInvalidValue;
    return launch_kernel(wmerge_tokens_kernel, dim3((n + 255) / 256, n_tok), dim3(256), 0, stream, pdl, parts, gates, y, n_parts, n, n_planes, plane_stride, resid, lids);
}

cudaError_t launch_scatter_rows(const float *x, uint32_t n_planes, size_t plane_stride, const uint32_t *table, const uint32_t *idx,
                                uint32_t list_stride, uint32_t col_off, uint32_t P, uint32_t n_groups, float *y, uint32_t n,
                                cudaStream_t stream) {
    if (n == 0 || n % 4 != 0 || plane_stride % 4 != 0 || P == 0 || n_groups == 0) return cudaErrorInvalidValue;
    scatter_rows_kernel<<<dim3((n + 1023) / 1024, P, n_groups), 256, 0, stream>>>(x, n_planes, plane_stride, table, idx, list_stride, col_off, y, n);
    return cudaGetLastError();
}

cudaError_t launch_group_by_expert(const uint32_t *lids, uint32_t n_pairs, uint32_t top_k, uint32_t n_local, uint32_t cap,
                                   uint32_t *cnt, uint32_t *tok_list, uint32_t *pair_list, uint32_t *table, cudaStream_t stream, bool pdl) {
    if (n_pairs == 0 || top_k == 0 || n_local == 0 || n_local > 256 || cap == 0) return cudaErrorInvalidValue;
    return launch_kernel(group_by_expert_kernel, dim3(1), dim3(32), 0, stream, pdl, lids, n_pairs, top_k, n_local, cap, cnt, tok_list, pair_list, table);
}

cudaError_t launch_nx_table(const uint32_t *cnt, uint32_t n_local, uint32_t col_off, uint32_t P, uint32_t *table, cudaStream_t stream) {
    nx_table_kernel<<<1, 32, 0, stream>>>(cnt, n_local, col_off, P, table);
    return cudaGetLastError();
}

cudaError_t launch_silu_mul(const float *gate, const float *up, float *h, uint32_t n, cudaStream_t stream) {
    silu_mul_kernel<<<(n + 255) / 256, 256, 0, stream>>>(gate, up, h, n);
    return cudaGetLastError();
}

cudaError_t launch_rope_append(const RopeAppendArgs &a, cudaStream_t stream) {
    if (a.head_dim == 0 || (a.head_dim & 1u)) return cudaErrorInvalidValue;
    const uint32_t half = a.head_dim / 2;
    const uint32_t n = ((a.q ? a.n_q_head : 0) + 2 * a.n_kv_head) * half;
    return launch_kernel(rope_append_kernel, dim3((n + 127) / 128, a.n_tok ? a.n_tok : 1), dim3(128), 0, stream, a.pdl != 0, a);
}

cudaError_t launch_rope_table(const int32_t *pos, float theta_scale, uint32_t head_dim, float2 *table, cudaStream_t stream,
                              uint32_t n_tok) {
    if (head_dim == 0 || (head_dim & 1u) || head_dim > 2048) return cudaErrorInvalidValue;
    rope_table_kernel<<<n_tok, head_dim / 2, 0, stream>>>(pos, theta_scale, head_dim / 2, table);
    return cudaGetLastError();
}

cudaError_t launch_argmax(const float *logits, uint32_t n, int32_t *out_idx, float *out_margin,
                          float *scratch, uint32_t *ticket, int sms, cudaStream_t stream, bool pdl, float *top3, uint32_t n_tok) {
    uint32_t grid = (n + 255) / 256;
    if (grid > (uint32_t)sms) grid = (uint32_t)sms;
    if (grid == 0) return cudaErrorInvalidValue;
    return launch_kernel(argmax_kernel, dim3(grid, n_tok), dim3(256), 0, stream, pdl, logits, n, out_idx, out_margin, scratch,
                         ticket, top3);
}

} // namespace flb
