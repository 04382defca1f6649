// Mixture-of-experts feed-forward block of the decode graph, single GPU or expert
// parallel over the GPUs of one box. Per token: router logits (f32 matvec),
// ROUTER_SEL (fl_op_router_sel, src/runtime/decode_params.h:234-265), the chosen
// experts' gate / up / down through the expert-indexed matvec (STREAM_DOT_IDX,
// src/runtime/runtime_internal.h:149-152) with the SiLU product between them, and
// WMERGE (fl_op_wmerge, :274-295); the reference builds the same chain as tasks
// (src/model/decoder.cpp:925-1045) and has no multi-GPU form.
//
// The tokens of a block are grouped by expert on the device (a stable counting sort of the (token, slot)
// pairs), and each of this rank's experts is walked ONCE per block: gate and up of all experts are one grouped
// multi-column matmul launch (matvec_tc_nx.cu) over the tokens that chose each expert, up to 16 per expert and pass, down
// is another, with the active experts and their token lists read on the device (an expert nobody chose costs
// nothing). The reference describes the same grouping for its task graph ("one tile set per
// DISTINCT expert serving every position that routed to it", src/model/decoder.cpp:927-930).
//
// Expert parallel: rank r of w holds experts [r * n / w, (r + 1) * n / w). The hidden states are
// replicated, so the dispatch half of the all-to-all moves nothing: every rank routes every token, runs
// only its own experts, merges with the other slots' gates set to zero, and the ranks' partial outputs
// are summed through peer memory by the exchange kernel of the tensor-parallel decoder (rank order, so
// every rank ends with identical bits). That sum is the combine half.
#include "capi_internal.h"

#include <algorithm>
#include <cstdlib>

using namespace flb;

struct fl_b200_moe {
    fl_b200_ctx *ctx = nullptr;
    fl_b200_moe_cfg c{};
    uint32_t rank = 0, world = 1, n_local = 0, base = 0;
    const float *router = nullptr;
    const uint8_t *wg = nullptr, *wu = nullptr, *wd = nullptr;
    float *logits = nullptr, *gates = nullptr, *mgates = nullptr, *part = nullptr, *partial = nullptr;
    uint32_t *ids = nullptr, *lids = nullptr, *tickets = nullptr;   // tickets: of the router's blocks, zero between launches
    uint32_t *cnt = nullptr, *tok_list = nullptr, *pair_list = nullptr;   // the pairs grouped by local expert (launch_group_by_expert)
    uint32_t *table = nullptr;                                            // active experts of a grouped launch
    // Used by one call at a time and written before it is read, hence shared by all blocks of a context (their calls are in order
    // on its stream): gate / up outputs and down outputs, planes of `rows` rows each, and the converted activations.
    std::shared_ptr<MoeScratch> scratch;
    float *g = nullptr, *u = nullptr, *d = nullptr, *h = nullptr;         // h: silu(gate) * up of every slot of one token
    uint8_t *xq = nullptr;
    uint32_t rows = 0, tgs = 0, planes_gu = 0, planes_d = 0;              // tgs: groups of four columns in xq
    bool expert_kernel = true;                                            // FLB_MOE_TOKEN=0 when it was created: a decoded token per slot
    uint8_t *arena = nullptr;                                             // the one allocation that holds the block's own buffers
    uint8_t *comm = nullptr;
    uint8_t *peers[kCommMaxRanks] = {};
    bool peers_set = false;
    uint32_t *comm_state = nullptr;
    // The launches of one forward call, recorded as a CUDA graph the second time a call repeats the
    // (x, y, n_tok) of the one before it, and replayed from then on (about 10 launches per token otherwise
    // cost more host time than the kernels take).
    struct { const float *x = nullptr; float *y = nullptr; uint32_t n_tok = 0; cudaGraph_t graph = nullptr; cudaGraphExec_t exec = nullptr; } rec;
};

namespace {

#define CKM(call)                                                      \
    do {                                                               \
        cudaError_t e_ = (call);                                       \
        if (e_ != cudaSuccess) return cuda_err(e_, #call);             \
    } while (0)

} // namespace

extern "C" {

int fl_b200_moe_create(fl_b200_ctx *ctx, const fl_b200_moe_cfg *cfg, uint32_t rank, uint32_t world, fl_b200_moe **out) {
    if (!ctx || !cfg || !out) return set_err(FL_B200_ERR_ARG, "moe_create: null pointer");
    const fl_b200_moe_cfg &c = *cfg;
    if (world == 0 || world > kCommMaxRanks || rank >= world) return set_err(FL_B200_ERR_ARG, "moe_create: rank %u of %u", rank, world);
    if (c.n_expert == 0 || c.n_expert > 256 || c.top_k == 0 || c.top_k > c.n_expert || c.n_expert % world)
        return set_err(FL_B200_ERR_ARG, "moe_create: %u experts, top %u, %u ranks", c.n_expert, c.top_k, world);
    if (c.n_embd % 256 || c.n_ff % 256 || c.n_embd < 512 || c.n_ff < 512 || c.max_tokens == 0)
        return set_err(FL_B200_ERR_ARG, "moe_create: n_embd and n_ff must be multiples of 256 (>= 512), max_tokens > 0");
    if (c.n_embd > 18432 || c.n_ff > 18432)
        return set_err(FL_B200_ERR_ARG, "moe_create: n_embd / n_ff above 18432 (the streaming matvec's column limit)");
    if (world > 1 && (c.n_embd > kCommMaxVec || c.n_embd % (4 * kCommChunks)))
        return set_err(FL_B200_ERR_ARG, "moe_create: n_embd %u does not fit the exchange buffer", c.n_embd);
    for (int fmt : {c.fmt_gate_up, c.fmt_down})
        if (fmt != FL_B200_Q4_K && fmt != FL_B200_Q6_K) return set_err(FL_B200_ERR_ARG, "moe_create: expert format %d (Q4_K or Q6_K)", fmt);
    CKM(cudaSetDevice(ctx->device));
    fl_b200_moe *m = new fl_b200_moe();
    if (const char *v = getenv("FLB_MOE_TOKEN")) m->expert_kernel = v[0] != '0';
    m->ctx = ctx; m->c = c; m->rank = rank; m->world = world;
    m->n_local = c.n_expert / world;
    m->base = rank * m->n_local;
    const size_t T = c.max_tokens, K = c.top_k, E = c.n_embd, F = c.n_ff;
    auto fail = [&](int rc) { fl_b200_moe_destroy(m); return rc; };
    auto alloc = [&](void **p, size_t bytes) -> int {
        if (cudaError_t e = cudaMalloc(p, bytes)) return cuda_err(e, "cudaMalloc (moe)");
        if (cudaError_t e = cudaMemsetAsync(*p, 0, bytes, ctx->stream)) return cuda_err(e, "cudaMemsetAsync (moe)");
        return FL_B200_OK;
    };
    // the most planes of partial results any number of tokens leads to (0: the per-slot form serves the shape)
    for (uint32_t P = 1; P <= kNxMaxTokens && P <= T; ++P) {
        const NxTensor gu{c.fmt_gate_up, nullptr, (uint32_t)F, 0, nullptr, 0, 0}, dn{c.fmt_down, nullptr, (uint32_t)E, 0, nullptr, 0, 0};
        const NxTensor two[2] = {gu, gu};
        const uint32_t a = matmul_tc_nx_parts(two, 2, c.n_embd, P, true), b = matmul_tc_nx_parts(&dn, 1, c.n_ff, P, true);
        if (a == 0 || b == 0) { m->planes_gu = m->planes_d = 0; break; }
        m->planes_gu = std::max(m->planes_gu, a);
        m->planes_d = std::max(m->planes_d, b);
    }
    const size_t n_gu = std::max(1u, m->planes_gu), n_d = std::max(1u, m->planes_d);
    // every active expert has at most 16 columns in a pass, all of them together at most one per pair
    m->tgs = (uint32_t)std::min<size_t>((size_t)m->n_local * (kNxMaxTokens / 4), T * K / 4 + std::min<size_t>(m->n_local, T * K));
    // Rows of the planes (the per-slot form: one slot at a time). Up to 16 tokens are one pass, a row per (token, slot) pair.
    // More of them go in passes of at most 16 columns per expert, whose rows are numbered through and added up to the pairs'
    // results after each: the planes don't grow with max_tokens.
    const size_t one_pass = std::min<size_t>(T, kNxMaxTokens) * K;
    m->rows = m->planes_gu == 0 ? 1 : (uint32_t)std::max(one_pass, std::min<size_t>(T * K, (size_t)m->n_local * kNxMaxTokens));
    const size_t R = m->rows, pairs = T > kNxMaxTokens || m->planes_gu == 0 ? T * K : K;   // (K: the per-slot form of one token)
    auto lay_out = [](const auto &bufs, uint8_t *at) {   // addresses from `at` on (nullptr: none); returns the bytes
        size_t total = 0;
        for (const auto &x : bufs) {
            if (at && x.bytes) *x.p = at + total;
            total += (x.bytes + 255) & ~(size_t)255;
        }
        return total;
    };
    struct Buf { void **p; size_t bytes; };
    const Buf shared[] = {{(void **)&m->g, n_gu * R * F * 4}, {(void **)&m->u, n_gu * R * F * 4}, {(void **)&m->d, m->planes_gu ? n_d * R * E * 4 : 0},
                          {(void **)&m->h, K * F * 4},
                          {(void **)&m->xq, m->planes_gu ? matmul_tc_nx_scratch_bytes((uint32_t)std::max(E, F), m->tgs, 1) : 0}};
    const size_t need = lay_out(shared, nullptr);
    m->scratch = ctx->moe_scratch.lock();
    if (!m->scratch || m->scratch->bytes < need) {
        m->scratch = std::make_shared<MoeScratch>();
        if (cudaError_t e = cudaMalloc((void **)&m->scratch->p, need)) return fail(cuda_err(e, "cudaMalloc (moe)"));
        m->scratch->bytes = need;
        ctx->moe_scratch = m->scratch;
    }
    lay_out(shared, m->scratch->p);
    // One allocation, zero-filled: the per-slot form leaves the part of a slot that is skipped as it was and multiplies it by gate 0.
    const Buf own[] = {
        {(void **)&m->logits, T * c.n_expert * 4}, {(void **)&m->tickets, T * 4}, {(void **)&m->gates, T * K * 4}, {(void **)&m->mgates, T * K * 4},
        {(void **)&m->ids, T * K * 4}, {(void **)&m->lids, T * K * 4}, {(void **)&m->table, (1 + (size_t)m->n_local) * 16},
        {(void **)&m->cnt, (size_t)m->n_local * 4}, {(void **)&m->tok_list, (size_t)m->n_local * T * 4},
        {(void **)&m->pair_list, (size_t)m->n_local * T * 4}, {(void **)&m->part, pairs * E * 4}, {(void **)&m->partial, world > 1 ? T * E * 4 : 0}};
    if (int rc = alloc((void **)&m->arena, lay_out(own, nullptr))) return fail(rc);
    lay_out(own, m->arena);
    if (world > 1) {   // mapped by the peers: allocations of their own
        if (int rc = alloc((void **)&m->comm, comm_buffer_bytes())) return fail(rc);
        if (int rc = alloc((void **)&m->comm_state, 64)) return fail(rc);
    }
    CKM(cudaStreamSynchronize(ctx->stream));
    *out = m;
    return FL_B200_OK;
}

void fl_b200_moe_destroy(fl_b200_moe *m) {
    if (!m) return;
    cudaSetDevice(m->ctx->device);
    cudaStreamSynchronize(m->ctx->stream);
    cudaFree(m->arena); cudaFree(m->comm); cudaFree(m->comm_state);
    if (m->rec.exec) cudaGraphExecDestroy(m->rec.exec);
    if (m->rec.graph) cudaGraphDestroy(m->rec.graph);
    delete m;
}

int fl_b200_moe_set_weights(fl_b200_moe *m, const float *router, const void *gate, const void *up, const void *down) {
    if (!m || !router || !gate || !up || !down) return set_err(FL_B200_ERR_ARG, "moe_set_weights: null pointer");
    if (((uintptr_t)gate | (uintptr_t)up | (uintptr_t)down | (uintptr_t)router) & 15u)
        return set_err(FL_B200_ERR_ARG, "moe_set_weights: tensors must be 16-byte aligned");
    m->router = router;
    m->wg = (const uint8_t *)gate; m->wu = (const uint8_t *)up; m->wd = (const uint8_t *)down;
    return FL_B200_OK;
}

int fl_b200_moe_comm(fl_b200_moe *m, void **buf, size_t *bytes) {
    if (!m || !buf || !bytes) return set_err(FL_B200_ERR_ARG, "moe_comm: null");
    *buf = m->comm;
    *bytes = m->comm ? comm_buffer_bytes() : 0;
    return FL_B200_OK;
}

int fl_b200_moe_set_peers(fl_b200_moe *m, void *const *bufs, uint32_t n) {
    if (!m || !bufs) return set_err(FL_B200_ERR_ARG, "moe_set_peers: null");
    if (n != m->world) return set_err(FL_B200_ERR_ARG, "moe_set_peers: %u buffers for %u ranks", n, m->world);
    for (uint32_t p = 0; p < n; ++p) {
        if (!bufs[p]) return set_err(FL_B200_ERR_ARG, "moe_set_peers: buffer of rank %u is null", p);
        m->peers[p] = (uint8_t *)bufs[p];
    }
    if (m->world > 1 && m->peers[m->rank] != m->comm) return set_err(FL_B200_ERR_ARG, "moe_set_peers: entry %u must be this rank's own buffer", m->rank);
    m->peers_set = true;
    return FL_B200_OK;
}

static RouterArgs moe_router_args(const fl_b200_moe *m, const float *x, uint32_t n_tok, const float *wnorm, float eps) {
    RouterArgs r{};
    r.router = m->router; r.x = x; r.n_embd = m->c.n_embd; r.n_expert = m->c.n_expert; r.wnorm = wnorm; r.eps = eps;
    r.logits = m->logits; r.tickets = m->tickets; r.ids = m->ids; r.gates = m->gates; r.lids = m->lids; r.mgates = m->mgates;
    r.n_tok = n_tok; r.top_k = m->c.top_k; r.norm = m->c.norm; r.scale = m->c.scale; r.base = m->base; r.n_local = m->n_local;
    return r;
}

// Shapes that the grouped form does not take.
static bool moe_per_slot(const fl_b200_moe *m) { return m->planes_gu == 0; }

static int moe_enqueue(fl_b200_moe *m, const float *x, uint32_t n_tok, float *y, bool per_slot, const float *wnorm = nullptr,
                       float eps = 0.f, const float *resid = nullptr);

int fl_b200_moe_forward(fl_b200_moe *m, const float *x, uint32_t n_tok, float *y) {
    if (!m || !x || !y) return set_err(FL_B200_ERR_ARG, "moe_forward: null pointer");
    if (!m->router) return set_err(FL_B200_ERR_STATE, "moe_forward: set the weights first");
    if (m->world > 1 && !m->peers_set) return set_err(FL_B200_ERR_STATE, "moe_forward: set the peers' exchange buffers first");
    if (n_tok == 0 || n_tok > m->c.max_tokens) return set_err(FL_B200_ERR_ARG, "moe_forward: %u tokens outside 1..%u", n_tok, m->c.max_tokens);
    cudaStream_t s = m->ctx->stream;
    CKM(cudaSetDevice(m->ctx->device));
    auto &rec = m->rec;
    const bool same = rec.x == x && rec.y == y && rec.n_tok == n_tok;
    if (same && rec.exec) {
        CKM(cudaGraphLaunch(rec.exec, s));
        return FL_B200_OK;
    }
    if (rec.exec) { cudaGraphExecDestroy(rec.exec); rec.exec = nullptr; }
    if (rec.graph) { cudaGraphDestroy(rec.graph); rec.graph = nullptr; }
    if (!same) {   // first sight of this call: run it directly
        rec.x = x; rec.y = y; rec.n_tok = n_tok;
        return moe_enqueue(m, x, n_tok, y, moe_per_slot(m));
    }
    CKM(cudaStreamBeginCapture(s, cudaStreamCaptureModeThreadLocal));
    const int rc = moe_enqueue(m, x, n_tok, y, moe_per_slot(m));
    cudaGraph_t g = nullptr;
    const cudaError_t e = cudaStreamEndCapture(s, &g);
    if (rc) { if (g) cudaGraphDestroy(g); return rc; }
    CKM(e);
    rec.graph = g;
    CKM(cudaGraphInstantiate(&rec.exec, g, 0));
    CKM(cudaGraphLaunch(rec.exec, s));
    return FL_B200_OK;
}

} // extern "C"

// One gate | up launch and one down launch per (token, slot) through the expert-indexed one-column matvec: the form
// for shapes the multi-column matmul does not take (rows that are not 16-byte pitched, e.g. Q6_K with 1024 columns).
// wnorm / resid (one GPU, inside a decoder step): x is the raw hidden state, normed on the fly by the router kernel
// and by the gate | up launch's prologue, and y = resid + the block's output (the merge's add1 term).
static int moe_enqueue_per_slot(fl_b200_moe *m, const float *x, uint32_t n_tok, float *y, const float *wnorm = nullptr,
                                float eps = 0.f, const float *resid = nullptr) {
    fl_b200_ctx *ctx = m->ctx;
    cudaStream_t s = ctx->stream;
    const fl_b200_moe_cfg &c = m->c;
    const uint32_t E = c.n_embd, F = c.n_ff, K = c.top_k;
    const uint64_t stride_gu = (uint64_t)F * row_bytes(c.fmt_gate_up, E), stride_d = (uint64_t)E * row_bytes(c.fmt_down, F);
    CKM(launch_router(moe_router_args(m, x, n_tok, wnorm, eps), s));
    const uint32_t rows_gu = (uint32_t)(stride_gu / row_bytes(c.fmt_gate_up, E)), rows_d = (uint32_t)(stride_d / row_bytes(c.fmt_down, F));
    static const int kMoePdl = getenv("FLB_MOE_PDL") ? atoi(getenv("FLB_MOE_PDL")) : 1;
    bool first_launch = true;
    const bool down_streams = matvec_is_streaming(c.fmt_down, F) && row_bytes(c.fmt_down, F) % 16 == 0;
    for (uint32_t t = 0; t < n_tok; ++t) {
        const float *xt = x + (size_t)t * E;
        for (uint32_t k = 0; k < K; ++k) {
            const uint32_t *lid = m->lids + (size_t)t * K + k;
            {   // gate and up of the slot's expert in one launch (both tensors carry the same id)
                MatvecArgs a{};
                a.n_tensors = 2;
                a.t[0] = {m->wg, m->g, nullptr, F, c.fmt_gate_up, 0, lid, rows_gu};
                a.t[1] = {m->wu, m->u, nullptr, F, c.fmt_gate_up, 0, lid, rows_gu};
                a.x = xt; a.cols = E; a.x_mode = MV_X_PLAIN; a.status = ctx->status;
                if (wnorm) { a.x_mode = MV_X_RMSNORM; a.wnorm = wnorm; a.eps = eps; }
                // Programmatic dependent launch from the second matvec launch on: the first one is an ordinary
                // dependent of the kernel that wrote the expert ids, and every later launch starts after it did,
                // so the ids (read at kernel entry, before the dependency wait) are in place for all of them.
                a.pdl = first_launch ? 0 : kMoePdl;
                a.expert_ids_ready = first_launch ? 0 : 1;
                first_launch = false;
                CKM(launch_matvec(a, ctx->sms, s));
            }
            {   // down, with silu(g) * u built while the activation is loaded (the streaming kernel's prologue;
                // rows that are not 16-byte pitched go through the generic kernel after a separate SiLU launch)
                MatvecArgs a{};
                a.n_tensors = 1;
                a.t[0] = {m->wd, m->part + ((size_t)t * K + k) * E, nullptr, E, c.fmt_down, 0, lid, rows_d};
                a.x = m->g; a.x2 = m->u; a.cols = F; a.x_mode = MV_X_SILU_MUL; a.status = ctx->status;
                a.pdl = kMoePdl;
                a.expert_ids_ready = 1;
                if (!down_streams) {
                    CKM(launch_silu_mul(m->g, m->u, m->g, F, s));
                    a.x2 = nullptr; a.x_mode = MV_X_PLAIN; a.pdl = 0;
                }
                CKM(launch_matvec(a, ctx->sms, s));
            }
        }
        float *dst = (m->world > 1 ? m->partial : y) + (size_t)t * E;
        CKM(launch_wmerge(m->part + (size_t)t * K * E, m->mgates + (size_t)t * K, m->world > 1 || !resid ? nullptr : resid + (size_t)t * E, nullptr, dst, 1.0f, K, E, K, s));
    }
    if (m->world > 1) {
        for (uint32_t t = 0; t < n_tok; ++t) {   // the combine: sum of the ranks' partial outputs, rank order
            AllReduceArgs r{};
            for (uint32_t p = 0; p < m->world; ++p) r.peers[p] = m->peers[p];
            r.in = m->partial + (size_t)t * E; r.resid = nullptr; r.out = y + (size_t)t * E; r.n = E;
            r.rank = m->rank; r.world = m->world; r.st = CommState{m->comm_state}; r.status = ctx->status; r.wait_ns = ctx->wait_limit_ns;
            CKM(launch_allreduce_resid(r, s, false));
        }
    }
    return FL_B200_OK;
}

// One token of a decoder step: the experts of all its slots in one launch for gate | up and one for down (matvec_expert.cu).
static bool moe_one_token(const fl_b200_moe *m) {
    const fl_b200_moe_cfg &c = m->c;
    return m->expert_kernel && m->world == 1 && c.top_k <= (uint32_t)m->ctx->sms && matvec_expert_takes(c.fmt_gate_up, c.n_embd, c.n_ff, c.top_k, c.n_expert) &&
           matvec_expert_takes(c.fmt_down, c.n_ff, c.n_embd, c.top_k, c.n_expert);
}

static int moe_enqueue_one_token(fl_b200_moe *m, const float *x, float *y, const float *wnorm, float eps, const float *resid) {
    cudaStream_t s = m->ctx->stream;
    const fl_b200_moe_cfg &c = m->c;
    static const int pdl = getenv("FLB_MOE_PDL") ? atoi(getenv("FLB_MOE_PDL")) : 1;
    RouterArgs r = moe_router_args(m, x, 1, wnorm, eps);
    r.pdl = pdl;
    CKM(launch_router(r, s));
    ExpertArgs e{};
    e.n_experts = c.n_expert; e.n_slots = c.top_k; e.id = m->lids; e.status = m->ctx->status; e.pdl = pdl;
    e.fmt = c.fmt_gate_up; e.w[0] = m->wg; e.w[1] = m->wu; e.rows = c.n_ff; e.cols = c.n_embd;
    // the router starts its dependents after it has waited for what lies in front of it, which wrote x
    e.x = x; e.wnorm = wnorm; e.eps = eps; e.y = m->h; e.x_ready = 1;
    CKM(launch_matvec_expert(e, m->ctx->sms, s));
    e.fmt = c.fmt_down; e.w[0] = m->wd; e.w[1] = nullptr; e.rows = c.n_embd; e.cols = c.n_ff;
    e.x = m->h; e.x_stride = c.n_ff; e.wnorm = nullptr; e.y = m->part; e.x_ready = 0;
    CKM(launch_matvec_expert(e, m->ctx->sms, s));
    CKM(launch_wmerge(m->part, m->mgates, resid, nullptr, y, 1.0f, c.top_k, c.n_embd, c.top_k, s, pdl != 0));
    return FL_B200_OK;
}

// the multi-column launches of the block as programmatic dependents of one another (FLB_MOE_PDL=0: plain launches)
static const int kMoePdlNx = getenv("FLB_MOE_PDL") ? atoi(getenv("FLB_MOE_PDL")) : 1;

// per_slot: the per-slot form. wnorm / resid (one GPU): x is the raw hidden state, normed inside the router kernel and the
// gate | up conversion, and y = resid + the block's output.
static int moe_enqueue(fl_b200_moe *m, const float *x, uint32_t n_tok, float *y, bool per_slot, const float *wnorm, float eps,
                       const float *resid) {
    fl_b200_ctx *ctx = m->ctx;
    cudaStream_t s = ctx->stream;
    const fl_b200_moe_cfg &c = m->c;
    const uint32_t E = c.n_embd, F = c.n_ff, K = c.top_k, T = c.max_tokens;
    if (per_slot) return moe_enqueue_per_slot(m, x, n_tok, y, wnorm, eps, resid);
    RouterArgs r = moe_router_args(m, x, n_tok, wnorm, eps);
    r.pdl = kMoePdlNx; r.w_after = wnorm ? 0 : 1;   // (a block called by itself: its router may have been written just before)
    CKM(launch_router(r, s));
    CKM(launch_group_by_expert(m->lids, n_tok * K, K, m->n_local, T, m->cnt, m->tok_list, m->pair_list, m->table, s, kMoePdlNx != 0));
    // Every local expert once for up to 16 of the tokens that chose it. The table and the lists live on the device, so the
    // launch sequence is the same for every routing (and can be replayed as a graph).
    const uint32_t P = std::min(n_tok, kNxMaxTokens);   // every pass is cut into the same parts, the last one too
    const bool one_pass = n_tok <= kNxMaxTokens;
    const size_t R = m->rows;
    const NxTensor gu[2] = {{c.fmt_gate_up, m->wg, F, 0, m->g, F, R * F}, {c.fmt_gate_up, m->wu, F, 0, m->u, F, R * F}};
    const NxTensor dn{c.fmt_down, m->wd, E, 0, m->d, E, R * E};   // down: the column of pair p is silu(g[p]) * u[p]
    const uint32_t parts_gu = matmul_tc_nx_parts(gu, 2, E, P, true), parts_d = matmul_tc_nx_parts(&dn, 1, F, P, true);
    for (uint32_t off = 0; off < n_tok; off += kNxMaxTokens) {
        if (off) CKM(launch_nx_table(m->cnt, m->n_local, off, P, m->table, s));
        NxIn in{};
        in.x = x; in.xstride = E; in.wnorm = wnorm; in.eps = eps;
        in.table = m->table; in.col_idx = m->tok_list; in.out_idx = one_pass ? m->pair_list : nullptr; in.list_stride = T; in.col_off = off;
        in.n_groups = std::min(m->n_local, n_tok * K); in.n_experts = m->n_local; in.sms = ctx->sms;
        in.n_tgs = std::min(in.n_groups * ((P + 3) / 4), n_tok * K / 4 + in.n_groups);
        // a conversion starts its dependent after it has waited for the kernel that wrote the table, so that the table is in place for
        // every matmul
        in.table_ready = kMoePdlNx; in.dep_first = 1;
        CKM(launch_nx_convert(in, gu, 1, E, P, m->xq, m->tgs, s, kMoePdlNx != 0));
        CKM(launch_nx_matmul(in, gu, 2, E, P, 0, m->xq, m->tgs, ctx->status, ctx->sms, s, kMoePdlNx != 0, true));
        in.x = m->g; in.x2 = m->u; in.xstride = F; in.wnorm = nullptr;
        in.n_parts = parts_gu; in.part_stride = R * F;
        in.col_idx = in.out_idx;
        // this conversion releases its dependent at entry: gate | up started after the conversion in front of it had waited, so that table
        // and weights are in place, and the down matmul's CTAs request weights as those of gate | up leave (2048 x 2048, 4 experts, one
        // token: 26.7 -> 24.6 us; 4096 x 6144, 16 experts, 12 tokens: 120.9 -> 120.1)
        in.dep_first = 0;
        CKM(launch_nx_convert(in, &dn, 1, F, P, m->xq, m->tgs, s, kMoePdlNx != 0));
        CKM(launch_nx_matmul(in, &dn, 1, F, P, 0, m->xq, m->tgs, ctx->status, ctx->sms, s, kMoePdlNx != 0, true));
        if (!one_pass) CKM(launch_scatter_rows(m->d, parts_d, R * E, m->table, m->pair_list, T, off, P, in.n_groups, m->part, E, s));
    }
    // WMERGE of every token: y[t] = sum_k gate[t][k] * part[t][k], slots of experts held elsewhere left out
    CKM(launch_wmerge_tokens(one_pass ? m->d : m->part, m->mgates, m->world > 1 ? m->partial : y, K, E, n_tok, s, one_pass ? parts_d : 1, R * E,
                             m->world > 1 ? nullptr : resid, m->world > 1 ? m->lids : nullptr, kMoePdlNx != 0 && one_pass));
    if (m->world > 1) {
        for (uint32_t t = 0; t < n_tok; ++t) {   // the combine: sum of the ranks' partial outputs, rank order
            AllReduceArgs r{};
            for (uint32_t p = 0; p < m->world; ++p) r.peers[p] = m->peers[p];
            r.in = m->partial + (size_t)t * E; r.resid = nullptr; r.out = y + (size_t)t * E; r.n = E;
            r.rank = m->rank; r.world = m->world; r.st = CommState{m->comm_state}; r.status = ctx->status; r.wait_ns = ctx->wait_limit_ns;
            CKM(launch_allreduce_resid(r, s, false));
        }
    }
    return FL_B200_OK;
}

int flb::moe_enqueue_tokens(fl_b200_moe *m, const float *x, uint32_t n_tok, float *y, uint32_t *n_launch, const float *wnorm,
                            float eps, const float *resid) {
    if (!m || !m->router || !m->wg) return set_err(FL_B200_ERR_STATE, "moe: weights not set");
    if (n_tok == 0 || n_tok > m->c.max_tokens) return set_err(FL_B200_ERR_ARG, "moe: %u tokens outside 1..%u", n_tok, m->c.max_tokens);
    const fl_b200_moe_cfg &c = m->c;
    if (m->world > 1 && (wnorm || resid)) return set_err(FL_B200_ERR_ARG, "moe: the fused norm / residual form is for one GPU");
    // One token inside a decoder step: the slots' experts through the one-column kernel (whole Mixtral-8x7B-shape step: 2.28 ms;
    // a launch per slot on the streaming kernel, which stays for the shapes the other does not take, 3.66, grouped 3.69); its
    // activation has 21 bits, relative error 2.3e-6 against 3e-7 of the grouped form, which is why a block called by itself stays
    // on that (fl_b200_moe_forward).
    const bool per_slot = moe_per_slot(m) || n_tok == 1;
    if (n_tok == 1 && wnorm && moe_one_token(m)) {
        if (n_launch) *n_launch = 4;
        return moe_enqueue_one_token(m, x, y, wnorm, eps, resid);
    }
    if (n_launch) {   // as moe_enqueue / moe_enqueue_per_slot enqueue them
        const bool down_streams = matvec_is_streaming(c.fmt_down, c.n_ff) && row_bytes(c.fmt_down, c.n_ff) % 16 == 0;
        const uint32_t passes = (n_tok + kNxMaxTokens - 1) / kNxMaxTokens;
        *n_launch = (!per_slot ? 2 + 4 * passes + (passes > 1 ? 2 * passes - 1 : 0) + 1 : 1 + n_tok * (c.top_k * (down_streams ? 2u : 3u) + 1)) + (m->world > 1 ? n_tok : 0u);
    }
    return moe_enqueue(m, x, n_tok, y, per_slot, wnorm, eps, resid);
}
fl_b200_ctx *flb::moe_ctx(const fl_b200_moe *m) { return m->ctx; }
const fl_b200_moe_cfg *flb::moe_cfg(const fl_b200_moe *m) { return &m->c; }
uint32_t flb::moe_world(const fl_b200_moe *m) { return m->world; }
uint64_t flb::moe_bytes_per_token(const fl_b200_moe *m) {
    const fl_b200_moe_cfg &c = m->c;
    return (uint64_t)c.n_expert * c.n_embd * 4 +
           (uint64_t)c.top_k * (2ull * c.n_ff * row_bytes(c.fmt_gate_up, c.n_embd) + (uint64_t)c.n_embd * row_bytes(c.fmt_down, c.n_ff));
}

extern "C" {

int fl_b200_moe_routing(fl_b200_moe *m, uint32_t n_tok, uint32_t *ids_host, float *gates_host) {
    if (!m || n_tok == 0 || n_tok > m->c.max_tokens) return set_err(FL_B200_ERR_ARG, "moe_routing: bad argument");
    const size_t n = (size_t)n_tok * m->c.top_k;
    if (ids_host) if (int rc = fl_b200_download(m->ctx, ids_host, m->ids, n * 4)) return rc;
    if (gates_host) if (int rc = fl_b200_download(m->ctx, gates_host, m->gates, n * 4)) return rc;
    return FL_B200_OK;
}

} // extern "C"
