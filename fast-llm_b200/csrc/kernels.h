// Internal launch interface between the C ABI (capi.cu), the decoder
// (decoder.cu) and the kernel translation units.
#pragma once
#include <cuda.h>
#include <cuda_runtime.h>
#include <stdint.h>

namespace flb {

// ---- dequant.cu ---------------------------------------------------------
cudaError_t launch_dequant(int fmt, const void *w, uint64_t rows, uint32_t cols, float *out, int sms,
                           cudaStream_t stream);

// ---- matvec.cu ----------------------------------------------------------
// One weight tensor of a (possibly multi-tensor) matvec launch. All tensors of
// a launch share the activation vector and the column count.
struct MatvecTensor {
    const uint8_t *w;     // packed rows, GGUF block layout, 16-byte aligned
    float *y;             // rows outputs
    const float *resid;   // optional: y[r] = resid[r] + dot   (nullptr: none)
    uint32_t rows;
    int fmt;
    uint32_t pitch;       // bytes between rows; 0 = packed (row_bytes(fmt, cols)). A column slice of a Q6_K
                          // tensor is stored with its rows zero-padded to a multiple of 16 bytes.
    // Expert indirection (STREAM_DOT_IDX, fl_idx_w, src/runtime/runtime_internal.h:149-152): the rows used
    // are those of expert *expert_id, expert_rows rows further down per expert (nullptr: none).
    // *t[0].expert_id == kExpertSkip: the whole launch reads nothing and leaves y as it is (expert
    // parallelism: the expert lives on another GPU). The id is read at kernel entry, so such a launch is not
    // made a programmatic dependent of the kernel that writes the id.
    const uint32_t *expert_id;
    uint32_t expert_rows;
};
constexpr uint32_t kExpertSkip = 0xFFFFFFFFu;

enum : int {
    MV_X_PLAIN = 0,    // activation = x
    MV_X_RMSNORM = 1,  // activation = x * rsqrt(mean(x^2)+eps) * wnorm
    MV_X_SILU_MUL = 2, // activation = silu(x) * x2
};

struct MatvecArgs {
    MatvecTensor t[4];
    int n_tensors;
    const float *x;
    const float *x2;      // MV_X_SILU_MUL: the "up" vector
    const float *wnorm;   // MV_X_RMSNORM
    float eps;
    uint32_t cols;
    int x_mode;
    int accumulate;       // 1: y[r] += dot (STREAM_DOT semantics); 0: y[r] = dot (+ resid)
    int swiglu;           // 1: t[0] = gate, t[1] = up (same shape and format): t[0].y[r] = silu(gate_r . x) * (up_r . x)
    uint32_t *status;     // device status word
    float *xn_out;        // optional: CTA 0 also writes the activation it built (nullptr: no)
    int pdl;              // launch with programmatic dependent launch
    int w_after;          // with pdl: nothing is read before the dependency is met, the weights neither (the kernel before may write them)
    int issue_late;       // 1: request the first weight stages after the activation loads are in flight instead of
                          // before the dependency wait (for launches whose CTAs only become resident when the previous
                          // kernel's CTAs leave, so that nothing is gained by requesting early)
    unsigned long long *trace;   // optional 4-entry timeline record of this launch (diagnostics)
    uint32_t *grid_bar;          // chained launches (launch_matvec_tc_chain): two zeroed words of device memory, the
                                 // state of the grid-wide barrier; one launch at a time may use them
    int expert_ids_ready;        // 1: the expert ids were complete before the previous kernel started, so the first
                                 // weight stages are requested before the dependency wait, as for a plain tensor
    // Tensor parallel: the activation is the sum of the ranks' partial vectors that an exchange launch
    // (launch_allreduce_push) is delivering into this rank's exchange buffer, plus a residual:
    // x = xr_resid + sum_r recv[r]. The kernel waits (bounded) for the ranks' flags of the epoch the
    // push launch recorded, adds in rank order (identical bits on all ranks) and CTA 0 also stores the
    // sum to xr_out (the new residual stream). nullptr: x is read as usual.
    const uint8_t *xr_buf;
    const uint32_t *xr_epoch;    // kCommChunks epoch counters of this rank's push launches
    const float *xr_resid;
    float *xr_out;
    uint32_t xr_world;
};

// Streaming kernel (Q4_K / Q6_K, cols a multiple of 256 and >= 512, rows 16-byte pitched) or the generic
// kernel (every other supported shape). Returns cudaErrorInvalidValue for
// unsupported arguments.
// 2-D tiled TMA descriptor over a row-major array (rows x dim0 elements, row pitch stride_bytes).
cudaError_t tensor_map_2d(CUtensorMap *m, uint32_t elem_bytes, const void *base, uint64_t dim0, uint64_t rows,
                          uint64_t stride_bytes, uint32_t box0, uint32_t box_rows, bool swizzle128);
cudaError_t tensor_map_lines_swz(CUtensorMap *m, const void *base, uint64_t rows, uint64_t pitch, uint32_t box_lines,
                                 uint32_t box_rows);   // [rows][pitch / 128][128 bytes], 128-byte swizzle (matvec.cu)
cudaError_t launch_matvec(const MatvecArgs &a, int sms, cudaStream_t stream);
// Q4_K / Q6_K launches that qualify run on the tensor-core streaming kernel (matvec_tc.cu).
bool matvec_tc_eligible(const MatvecArgs &a);
cudaError_t launch_matvec_tc(const MatvecArgs &a, int sms, cudaStream_t stream);
// n (1..4) matvecs in ONE launch, each consuming what the one before it wrote (O -> gate|up -> down -> next Q/K/V),
// with grid-wide barriers in between and the weights of the next phase streaming meanwhile. cudaErrorNotSupported
// when a phase does not qualify: launch them one by one then. args[0].grid_bar names the barrier state.
cudaError_t launch_matvec_tc_chain(const MatvecArgs *args, int n, int sms, cudaStream_t stream);
cudaError_t matvec_tc_init(void);
// The experts that one token selected (matvec_expert.cu), slot k's being id[k]: y[k * rows + r] = silu(gate_r . h) * (up_r . h) with
// h = RMSNorm(x) * wnorm (w[1] set), or y[k * rows + r] = w_r . (x + k * x_stride). The bits of a streaming launch per slot (gate | up: up to
// 6144 columns).
struct ExpertArgs {
    int fmt;
    const void *w[2];            // gate and up, or down and nullptr: the experts' rows one behind the other, packed
    uint32_t rows, cols, n_experts, n_slots;   // rows: of one expert
    const uint32_t *id;          // device; gate | up: from the launch in front; down: in place before the launch in front read anything
    const float *x, *wnorm;
    uint32_t x_stride;
    float eps, *y;
    int x_ready;                 // x was complete before the launch in front started its dependents
    uint32_t *status;
    int pdl;
};
bool matvec_expert_takes(int fmt, uint32_t cols, uint32_t rows, uint32_t n_slots, uint32_t n_experts);
cudaError_t launch_matvec_expert(const ExpertArgs &e, int sms, cudaStream_t stream);
cudaError_t matvec_expert_init(void);
// Several activation columns (P <= 16) in one pass over up to three Q4_K / Q6_K / Q8_0 tensors on the tensor cores
// (matvec_tc_nx.cu): y[p * ystride + r] (+)= dot(W[r], column p). Two launches: launch_nx_convert builds the activation's
// operand image(s) in xq, launch_nx_matmul walks the weights.
constexpr uint32_t kNxMaxTokens = 16, kNxMaxCols = 18432;
constexpr uint32_t kMaxPlanes = 9;   // planes of partial results that the next conversion adds: no form may leave more
constexpr uint32_t kAttnRecord = 132;   // floats of one split's record of one query head: context[128], maximum, sum, pad
struct NxTensor {
    int fmt;
    const void *w;           // rows x cols, GGUF block layout (grouped: the experts' slices one behind the other)
    uint32_t rows, pitch;    // pitch 0 = packed rows
    float *y;                // output row blocks, ystride floats apart
    uint32_t ystride;
    size_t part_stride;      // floats between the planes of partial results (matmul_tc_nx_parts > 1)
};
struct NxIn {
    const float *x;          // column p: row p, xstride floats apart
    const float *x2;         // optional: the column is SiLU(x) * x2 (same strides)
    uint32_t xstride, n_parts;   // n_parts planes of x (and x2), part_stride floats apart, are added in order (0 = 1)
    size_t part_stride;
    const float *resid;      // optional: + resid (row p, rstride apart)
    float *x_out;            // optional: the sum is stored here too (row p, rstride apart)
    uint32_t rstride;
    const float *wnorm;      // optional: RMSNorm(column) * wnorm; the matmul applies the 1 / rms to its results
    float eps;
    const float *att;        // optional, in place of x: the columns are the attention contexts of heads of 128 whose splits'
    uint32_t n_splits;       // records (launch_attn_decode with records_only) are added up here
    // Grouped columns (mixture of experts): `table` (launch_nx_table) lists the active experts; column p of an expert is row
    // col_idx[expert * list_stride + col_off + p] of x and goes to output row block out_idx[the same]. Without col_idx / out_idx
    // the rows are numbered through, expert by expert in the table's order.
    const uint32_t *table, *col_idx, *out_idx;
    uint32_t list_stride, col_off, n_groups, n_experts, n_tgs;   // n_groups: upper bound of active experts; n_tgs: of their groups of four columns
    uint32_t sms;            // of the device
    int table_ready;         // 1: the table was complete before the kernel in front of the matmul started
    int dep_first;           // 1: the launch after the conversion starts only when what lies in front of the conversion has completed
    int tm;                  // 1: launch_nx_convert builds the image of matmul_tm.cu (Q4_K or Q6_K, one format, not grouped)
};
// Number of parts the columns are cut into (1: y is the result; more: planes of partial sums); 0: not taken. split: planes cost the
// caller nothing extra, cut as finely as is best.
// tm_sms > 0: launches that matmul_tm_takes on so many SMs are cut as that form cuts them.
uint32_t matmul_tc_nx_parts(const NxTensor *t, int n, uint32_t cols, uint32_t P, bool split = false, int tm_sms = 0);
// tgs: groups of four columns in the image(s) (grouped: of all active experts together)
size_t matmul_tc_nx_scratch_bytes(uint32_t cols, uint32_t tgs, int layouts);
// n = 0 tensors: only x_out is written. cudaErrorNotSupported: strides or addresses the vector loads do not take.
cudaError_t launch_nx_convert(const NxIn &in, const NxTensor *t, int n, uint32_t cols, uint32_t P, uint8_t *xq, uint32_t tgs_cap,
                              cudaStream_t stream, bool pdl);
cudaError_t launch_nx_matmul(const NxIn &in, const NxTensor *t, int n, uint32_t cols, uint32_t P, int accumulate, const uint8_t *xq,
                             uint32_t tgs_cap, uint32_t *status, int sms, cudaStream_t stream, bool pdl, bool split = false);
cudaError_t launch_reduce_parts(const float *part, size_t part_stride, uint32_t n_parts, float *y, uint32_t rows, uint32_t ystride,
                                uint32_t P, int accumulate, cudaStream_t stream, bool pdl);
// The table of a grouped launch: of cnt[e] listed columns of expert e those from col_off on, at most P.
cudaError_t launch_nx_table(const uint32_t *cnt, uint32_t n_local, uint32_t col_off, uint32_t P, uint32_t *table, cudaStream_t stream);
// The same on tcgen05, weights and results in tensor memory (matmul_tm.cu): Q4_K or Q6_K, one format, not grouped; between launch_nx_convert with
// in.tm set and the next conversion or reduction, as launch_nx_matmul. The image of 256 columns takes 8512 bytes up to 8 tokens,
// else 17024: less than matmul_tc_nx_scratch_bytes provides.
bool matmul_tm_takes(const NxTensor *t, int n, uint32_t cols, uint32_t P, int sms);   // launches with planes (split) for which it is the faster form
bool matmul_tm_takes_whole(const NxTensor *t, int n, uint32_t cols, uint32_t P, int sms);   // and without
uint32_t matmul_tm_parts(const NxTensor *t, int n, uint32_t cols, bool split, int sms);
cudaError_t launch_tm_matmul(const NxIn &in, const NxTensor *t, int n, uint32_t cols, uint32_t P, int accumulate, const uint8_t *xq,
                             uint32_t *status, int sms, cudaStream_t stream, bool pdl, bool split);
cudaError_t matmul_tm_init(void);
// FLB_UMMA in the environment now (-1: not set). 1: every Q4_K call of several columns on that form, whole tiles; 2: every Q4_K and
// Q6_K call, with planes as in a batch pass; 0: no launch of a batch pass on it.
int matmul_tm_switch(void);
cudaError_t matmul_tc_nx_init(void);
// True when launch_matvec would take the streaming kernel for this shape.
bool matvec_is_streaming(int fmt, uint32_t cols);
// Dynamic shared memory the streaming kernel needs for (cols, formats used).
size_t matvec_smem_bytes(uint32_t cols, bool use_q4k, bool use_q6k, int *stages_out, int *warps_out, bool use_q8_0 = false);
// [p, p + bytes) lies in one allocation of `device` (false: elsewhere, or unknown).
bool in_device_memory(int device, const void *p, size_t bytes);
cudaError_t matvec_init(void);   // sets the dynamic shared memory attribute once

// ---- attn.cu ------------------------------------------------------------
struct AttnArgs {
    const float *q;        // [batch][n_q_head][128] f32 (post-RoPE unless rope fused)
    uint32_t q_stride;     // floats between the sequences' queries (0: n_q_head * 128)
    const __half *k;       // [batch][n_kv_head][kv_stride][128] f16
    const __half *v;       // same layout
    float *out;            // [batch][n_q_head][128]
    float *part;           // scratch: [batch][n_q_head][n_splits][132] (context[128], max, sum, pad)
    uint32_t *tickets;     // scratch: [batch][n_kv_head], zero before first use; self-resetting
    const int32_t *pos;    // device scalar: last valid position of sequence 0 (kv_len = *pos + 1); nullptr -> kv_len
    uint32_t kv_len;       // used when pos == nullptr
    uint32_t kv_len_step;  // sequence b attends kv_len + b * kv_len_step keys (draft verification: step 1)
    uint32_t shared_kv;    // 1: all sequences read the same cache (batch_stride ignored)
    uint32_t pos_stride;   // sequence b takes its position from pos[b * pos_stride] (0: all from pos[0]; independent sequences: 1)
    uint32_t kv_stride;    // positions allocated per head
    uint64_t batch_stride; // elements between sequences in k / v
    uint32_t n_q_head, n_kv_head, batch, n_splits;
    float scale;
    uint32_t *status;
    int pdl;
    int late;              // dependents are released behind the tiles instead of at entry (attn_release)
    int records_only;      // several positions of one cache (attn_uses_records): leave the splits' records in part, out is not written
    int per_position;      // several positions of one cache, but one CTA per position all the same (attn_few_tiles)
    unsigned long long *trace;   // optional 4-entry timeline record (diagnostics)
    // Fused RoPE + KV append (the decoder's launch plan): q arrives un-rotated; rope_k / rope_v are this
    // token's k and v ([batch][n_kv_head][128] f32, k un-rotated); the kernel rotates q and k by the angle
    // of position *pos and appends k, v (f16) at row *pos of k_append / v_append (the same arrays as k, v).
    float2 *lse_out;                // optional [batch][n_q_head]: (max score, sum of exp(score - max)) of each head
    const float *rope_k, *rope_v;   // nullptr: q is already rotated and the cache is complete
    __half *k_append, *v_append;
    float theta_scale;              // freq_base^(-2/128)
    const float2 *rope_table;       // optional: (cos, sin) of the 64 angles of position *pos, computed once per step
                                    // (launch_rope_table); nullptr: every CTA computes them itself
    CUtensorMap kmap, vmap;         // filled by attn_make_maps
};
cudaError_t attn_make_maps(AttnArgs &a);
// Positions over one cache so few and short that the one-position kernel, a single launch, is the faster one.
bool attn_few_tiles(uint32_t n_kv_head, uint32_t batch, uint32_t kv_len);
bool attn_uses_records(const AttnArgs &a);   // the launch is one of several positions over one cache (attn_shared_kernel)
cudaError_t launch_attn_decode(const AttnArgs &a, cudaStream_t stream);
void attn_release(AttnArgs &a, int sms);     // pdl and late of a call by itself (pos == nullptr), everything else set
// Same kernel with the split-KV scratch in a fixed file-scope device array
// (no allocation at call time); cudaErrorMemoryAllocation when the launch needs
// more than attn_static_max_records() records or attn_static_max_tickets()
// (KV head, sequence) pairs.
cudaError_t launch_attn_decode_static(AttnArgs a, int device, cudaStream_t stream, size_t *records_needed);
size_t attn_static_max_records(void);
uint32_t attn_static_max_tickets(void);
cudaError_t attn_init(void);
uint32_t attn_pick_splits(uint32_t n_kv_head, uint32_t batch, uint32_t kv_len, int sms, bool shared_kv = false);
uint32_t attn_used_splits(uint32_t n_splits, uint32_t kv_len);   // those of n_splits that hold keys when kv_len keys are cut
size_t attn_part_floats(uint32_t n_q_head, uint32_t batch, uint32_t n_splits);

// ---- comm.cu: exchange steps of the tensor-parallel step ----------------------
constexpr uint32_t kCommMaxRanks = 8;
constexpr uint32_t kCommMaxVec = 8192;     // floats per partial vector (hidden size)
constexpr uint32_t kCommChunks = 8;        // CTAs (and flags) per all-reduce
constexpr size_t kCommFlagsOff = (size_t)2 * kCommMaxRanks * kCommMaxVec * 4;
constexpr size_t kCommTopOff = kCommFlagsOff + (size_t)2 * kCommMaxRanks * kCommChunks * 4;
constexpr size_t kCommTFlagOff = kCommTopOff + (size_t)2 * kCommMaxRanks * 16;
constexpr size_t kCommBytes = kCommTFlagOff + (size_t)2 * kCommMaxRanks * 4;
struct CommState {
    uint32_t *epoch;   // kCommChunks + 1 device counters: epoch of the last exchange per chunk, then of the argmax exchange
};
struct AllReduceArgs {
    uint8_t *peers[kCommMaxRanks];   // every rank's communication buffer as mapped here; peers[rank] is local
    const float *in;                 // this rank's partial vector
    const float *resid;              // optional, added once (local)
    float *out;
    uint32_t n, rank, world;
    CommState st;
    uint32_t *status;
    uint64_t wait_ns;                // limit of the wait for the peers' flags (0 = one second)
};
struct TopExchangeArgs {
    uint8_t *peers[kCommMaxRanks];
    const float *top3;               // {best, index bits, runner-up} of this rank's slice
    uint32_t index_base;             // first global index of the slice
    int32_t *out_idx;
    float *out_margin;
    uint32_t rank, world;
    CommState st;
    uint32_t *status;
    uint64_t wait_ns;
};
// Sequence-parallel attention: every rank attended its slice of the keys and holds, per (sequence,
// query head) record, the normalised context and (max, sum); the exchange merges the ranks' records.
struct LseCombineArgs {
    uint8_t *peers[kCommMaxRanks];   // exchange buffers: [2 slots][world][max_records][132] f32, then flags [2][world][kLseChunks]
    const float *out_local;          // [n][128]
    const float2 *lse_local;         // [n]
    float *out;                      // [n][128]
    uint32_t n, max_records, rank, world;
    uint32_t *epoch;                 // kLseChunks device counters
    uint32_t *status;
    uint64_t wait_ns;                // limit of the wait for the peers' flags (0 = one second)
};
constexpr uint32_t kLseChunks = 32;
size_t lse_buffer_bytes(uint32_t max_records);
cudaError_t launch_lse_combine(const LseCombineArgs &a, cudaStream_t stream);
size_t comm_buffer_bytes(void);
cudaError_t launch_allreduce_resid(const AllReduceArgs &a, cudaStream_t stream, bool pdl);
// The push half alone (stores + flags; resid / out unused): the consumer matvec waits and adds.
cudaError_t launch_allreduce_push(const AllReduceArgs &a, cudaStream_t stream, bool pdl);
cudaError_t launch_argmax_exchange(const TopExchangeArgs &a, cudaStream_t stream, bool pdl);

// ---- glue.cu ------------------------------------------------------------
// dst[0 .. bytes) = value; dst of any alignment.
cudaError_t launch_fill(void *dst, int value, size_t bytes, int sms, cudaStream_t stream, bool pdl);
// rows vectors of n floats, `stride` floats apart in x and in y (one weight vector for all).
cudaError_t launch_rmsnorm(const float *x, const float *wnorm, float *y, float eps, uint32_t n,
                           cudaStream_t stream, uint32_t rows = 1, uint32_t stride = 0);
cudaError_t launch_add2(const float *a, const float *b, float *y, uint32_t n, cudaStream_t stream);
// Router of a block in one launch: logits[t][e] = dot(router[e], x[t]), and what launch_router_sel does, by a token's last block.
struct RouterArgs {
    const float *router, *x, *wnorm;   // [n_expert][n_embd]; [n_tok][n_embd]; optional: the logits are those of RMSNorm(x) * wnorm
    float eps;
    uint32_t n_embd, n_expert, n_tok;
    float *logits;                     // [n_tok][n_expert]
    uint32_t *tickets;                 // [n_tok], zero between launches
    uint32_t *ids, *lids;              // the rest: as launch_router_sel
    float *gates, *mgates;
    uint32_t top_k, norm;
    float scale;
    uint32_t base, n_local;
    int pdl, w_after;                  // w_after: with pdl, nothing is read before the dependency is met
};
cudaError_t launch_router(const RouterArgs &a, cudaStream_t stream);
// The (token, slot) pairs of a block, grouped by the local expert they chose (a stable counting sort: within an
// expert the pairs stay in ascending order): cnt[e] pairs for expert e, their tokens in tok_list[e * cap + i] and
// their pair indices (token * top_k + slot) in pair_list[e * cap + i]. lids: local expert of every pair or kExpertSkip. The table
// of a grouped launch over the first 16 of each (launch_nx_table).
cudaError_t launch_group_by_expert(const uint32_t *lids, uint32_t n_pairs, uint32_t top_k, uint32_t n_local, uint32_t cap,
                                   uint32_t *cnt, uint32_t *tok_list, uint32_t *pair_list, uint32_t *table, cudaStream_t stream, bool pdl);
// fl_op_router_sel (src/runtime/decode_params.h:234-265) for n_tok tokens in one launch (one warp per token):
// softmax over n_expert logits, top_k by weight; logits [n_tok][n_expert], ids / gates [n_tok][top_k]. Expert
// parallel (lids, mgates != nullptr): also the expert's index among this rank's experts [base, base + n_local)
// or the skip mark, and the gate or 0.
cudaError_t launch_router_sel(const float *logits, uint32_t *ids, float *gates, uint32_t n_tok, uint32_t n_expert, uint32_t top_k,
                              uint32_t norm, float scale, cudaStream_t stream, uint32_t *lids = nullptr,
                              float *mgates = nullptr, uint32_t base = 0, uint32_t n_local = 0);
// fl_op_wmerge (src/runtime/decode_params.h:274-295).
cudaError_t launch_wmerge(const float *parts, const float *gates, const float *add1, const float *add2, float *y,
                          float scale, uint32_t n_parts, uint32_t n, uint32_t n_full, cudaStream_t stream, bool pdl = false);
// fl_op_wmerge for n_tok tokens in one launch: y[t] = (resid[t] +) sum_q gates[t][q] * parts[t][q] (products and sums
// rounded in the reference's order); a part is the sum of n_planes planes, plane_stride floats apart.
cudaError_t launch_wmerge_tokens(const float *parts, const float *gates, float *y, uint32_t n_parts, uint32_t n, uint32_t n_tok,
                                 cudaStream_t stream, uint32_t n_planes = 1, size_t plane_stride = 0, const float *resid = nullptr,
                                 const uint32_t *lids = nullptr, bool pdl = false);   // lids: slots whose entry is kExpertSkip are left out
// Rows numbered through by a grouped launch's table (row r of x: n_planes planes of n floats, plane_stride apart) to the rows of
// y that their columns stand for: y[idx[expert * list_stride + col_off + p]] = the sum of the planes. n a multiple of 4.
cudaError_t launch_scatter_rows(const float *x, uint32_t n_planes, size_t plane_stride, const uint32_t *table, const uint32_t *idx,
                                uint32_t list_stride, uint32_t col_off, uint32_t P, uint32_t n_groups, float *y, uint32_t n,
                                cudaStream_t stream);
cudaError_t launch_silu_mul(const float *gate, const float *up, float *h, uint32_t n, cudaStream_t stream);
// RoPE (adjacent pairs) on q in place and on k, then store k and v as f16 at
// row *pos of a cache laid out [n_kv_head][kv_stride][head_dim].
struct RopeAppendArgs {
    float *q;              // [n_q_head][head_dim], rotated in place (nullptr: skip)
    const float *k;        // [n_kv_head][head_dim] (pre-RoPE)
    const float *v;        // [n_kv_head][head_dim]
    __half *kcache, *vcache;
    const int32_t *pos;
    uint32_t n_q_head, n_kv_head, head_dim, kv_stride;
    float theta_scale;     // freq_base^(-2/head_dim), computed on the host
    int pdl;
    // batch pass: n_tok tokens (0 = 1), token i at q + i * q_tok_stride, k / v + i * kv_tok_stride, position pos[i]
    uint32_t n_tok, q_tok_stride, kv_tok_stride;
    uint64_t seq_elems;    // independent sequences: token i appends to the cache of sequence i, seq_elems halves further (0: one cache)
    uint32_t n_planes;     // q, k and v are the sums of n_planes planes, plane_stride floats apart (0 = 1); the rotated q goes to the first
    uint64_t plane_stride;
    const float2 *table;   // optional: (cos, sin) of token i's angles, head_dim / 2 per token (launch_rope_table)
};
cudaError_t launch_rope_append(const RopeAppendArgs &a, cudaStream_t stream);
// (cos, sin) of pos * theta_scale^i, i < head_dim / 2, with the angle built by repeated multiplication exactly as
// fl_op_rope_ds2 does (src/runtime/decode_params.h:124-160); table: head_dim / 2 float2.
cudaError_t launch_rope_table(const int32_t *pos, float theta_scale, uint32_t head_dim, float2 *table, cudaStream_t stream,
                              uint32_t n_tok = 1);   // n_tok positions, one table row each
// Greedy argmax with the reference's tie rule (lowest index) and the
// top1 - top2 margin. out_idx: int32, out_margin: float; scratch: 2*blocks*2 floats.
cudaError_t launch_argmax(const float *logits, uint32_t n, int32_t *out_idx, float *out_margin,
                          float *scratch, uint32_t *ticket, int sms, cudaStream_t stream, bool pdl = false,
                          float *top3 = nullptr,    // top3: optional {best, index bits, runner-up}
                          uint32_t n_tok = 1);      // rows of logits (n apart); scratch, ticket, outputs and top3 per row
constexpr uint32_t kArgmaxScratch = 3 * 1024;   // floats of scratch per row
// Embedding row gather + dequant: out[i][0..cols) = dequant(table row token[i]), i < n_tok.
cudaError_t launch_embed(int fmt, const void *table, const int32_t *token, uint32_t cols, float *out,
                         cudaStream_t stream, bool pdl = false, uint32_t n_tok = 1);

} // namespace flb
