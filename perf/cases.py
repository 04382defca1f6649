"""The work this library is used for, as cases that can be timed and compared: what a program that decodes with a
k-quant Llama-shape model on one GPU calls, through the Python mirror of the C ABI (``fast_llm_b200``).

Families ("kind"):

  matvec     one STREAM_DOT: y += W x for 1..16 activation columns (Context.matvec), any weight format
  attention  decode attention of every query head over an f16 cache (Context.attn_decode)
  moe        one mixture-of-experts feed-forward block over 1..16 tokens (MoeBlock.forward)
  step       single-token decode steps of a whole model, each step's token fed to the next (Decoder.step)
  batch      several positions of one sequence in one pass (Decoder.step_batch): draft verification, prompt chunks
  seqs       several independent sequences in lock step (Decoder.seqs_step)

Sizes are those of the benchmark configurations (the 8B and the Mixtral-8x7B shape, 1024 to 128K keys) and generic
ones beside them. Weights are synthetic: random quants and scales in the GGUF block layouts, scaled to zero mean and a
standard deviation of 1 / sqrt(columns), so that activations keep unit size through the layers as in a trained model.
"""
import ctypes as C
import math
import random

import torch

from fast_llm_b200 import capi
from fast_llm_b200.decoder import Decoder
from fast_llm_b200.moe import MoeBlock

FMT = {"Q4_K": capi.Q4_K, "Q6_K": capi.Q6_K, "Q8_0": capi.Q8_0}
HEAD_DIM = 128
Q4_K_M = {"wq": "Q4_K", "wk": "Q4_K", "wv": "Q6_K", "wo": "Q4_K", "gate": "Q4_K", "up": "Q4_K", "down": "Q6_K",
          "output": "Q6_K", "tok_embd": "Q6_K"}
RECIPES = {"Q4_K_M": Q4_K_M, "Q4_K": {k: "Q4_K" for k in Q4_K_M}, "Q8_0": {k: "Q8_0" for k in Q4_K_M}}
LAYER = ("wq", "wk", "wv", "wo", "gate", "up", "down")
LLAMA_8B = dict(n_layer=32, n_embd=4096, n_kv_head=8, n_ff=14336, n_vocab=128256, recipe="Q4_K_M", rope_base=500000.0)
MIXTRAL = dict(n_layer=32, n_embd=4096, n_kv_head=8, n_ff=14336, n_vocab=32000, recipe="Q4_K_M", rope_base=1000000.0,
               n_expert=8, top_k=2)


def listed():
    return [
        # Latency: the smallest calls, one operator at a time (the task-level API's granularity).
        dict(name="matvec_q4k_4096", kind="matvec", fmt="Q4_K", rows=4096, cols=4096, nx=1),
        dict(name="attn_1k", kind="attention", n_kv_head=8, kv_len=1024, batch=1),
        # An 8-bit projection with a few draft columns, rows that are no multiple of anything.
        dict(name="matmul_q80_3col", kind="matvec", fmt="Q8_0", rows=11007, cols=4096, nx=3),
        # The FFN of the 8B shape over a verification batch: gate rows, 8 columns.
        dict(name="matmul_q4k_8col", kind="matvec", fmt="Q4_K", rows=14336, cols=4096, nx=8),
        # Long-context attention, a few requests with ragged length.
        dict(name="attn_64k_b4", kind="attention", n_kv_head=8, kv_len=65000, batch=4),
        # Mixture-of-experts block at the Mixtral shape, 16 tokens, top-2 of 8.
        dict(name="moe_block_16", kind="moe", n_embd=4096, n_ff=14336, n_expert=8, top_k=2, n_tok=16, fmt="Q4_K"),
        # A 3B-class model in 8-bit weights, a width that is no power of two, short context.
        dict(name="step_3b_q80", kind="step", n_layer=28, n_embd=3072, n_kv_head=6, n_ff=8192, n_vocab=32000, recipe="Q8_0",
             rope_base=500000.0, pos=777, n_step=4),
        # The headline: greedy decoding at the 8B shape, 8192 positions behind it.
        dict(name="step_8b_kv8192", kind="step", pos=8192, n_step=4, **LLAMA_8B),
        # Draft verification: 8 positions in one pass over 4096 cached ones.
        dict(name="verify_8b_k8", kind="batch", pos=4096, m=8, **LLAMA_8B),
        # Prompt ingestion in chunks: 16 positions in one pass, early in the prompt.
        dict(name="chunk_8b_16", kind="batch", pos=1001, m=16, **LLAMA_8B),
        # Serving: 16 independent sequences of different lengths, one token each.
        dict(name="seqs_8b_16", kind="seqs", pos=4096, n_seq=16, **LLAMA_8B),
        # Greedy decoding of a whole mixture-of-experts model (Mixtral-8x7B shape).
        dict(name="step_moe_kv4096", kind="step", pos=4096, n_step=2, **MIXTRAL),
    ]


def _log(rng, lo, hi):
    return int(round(math.exp(rng.uniform(math.log(lo), math.log(hi)))))


def _model(rng, max_layer):
    recipe = rng.choice(["Q4_K_M", "Q4_K_M", "Q4_K", "Q8_0"])
    # the decoder takes Q6_K rows of whole 16-byte pieces: widths that are multiples of 2048
    kv, n_ff = rng.randint(2, 8), 256 * rng.randint(16, 56)
    if recipe == "Q4_K_M":
        kv, n_ff = rng.choice([4, 8]), 2048 * rng.randint(2, 7)
    return dict(n_layer=rng.randint(2, max_layer), n_embd=512 * kv, n_kv_head=kv, n_ff=n_ff, n_vocab=_log(rng, 8000, 128256),
                recipe=recipe, rope_base=500000.0)


def draw(rng):
    kind = rng.choice(["matvec", "matvec", "attention", "attention", "moe", "step", "batch", "seqs"])
    if kind == "matvec":
        return dict(kind=kind, fmt=rng.choice(["Q4_K", "Q6_K", "Q8_0"]), rows=_log(rng, 256, 131072),
                    cols=256 * _log(rng, 2, 56), nx=rng.choice([1, 1, rng.randint(2, 16)]))
    if kind == "attention":
        kv_len = _log(rng, 64, 131072)
        return dict(kind=kind, n_kv_head=rng.choice([2, 4, 8, 8]), kv_len=kv_len, batch=rng.randint(1, 16))
    if kind == "moe":
        return dict(kind=kind, n_embd=2048 * rng.randint(1, 2), n_ff=2048 * rng.randint(1, 7), n_expert=rng.choice([4, 8, 16]),
                    top_k=rng.randint(1, 4), n_tok=rng.randint(1, 16), fmt=rng.choice(["Q4_K", "Q4_K", "Q6_K"]))
    if kind == "step":
        return dict(kind=kind, pos=_log(rng, 16, 16384), n_step=4, **_model(rng, 16))
    if kind == "batch":
        return dict(kind=kind, pos=_log(rng, 16, 8192), m=rng.randint(2, 16), **_model(rng, 16))
    return dict(kind=kind, pos=_log(rng, 16, 4096), n_seq=rng.randint(2, 16), **_model(rng, 16))


# ---- inputs ----------------------------------------------------------------------------------------------------

_CTX = []


def _context():
    """One library context per process, as in a program that uses the library."""
    if not _CTX:
        _CTX.append(capi.Context(0))
    return _CTX[0]


def _gen(seed):
    g = torch.Generator(device="cuda")
    g.manual_seed(int(seed))
    return g


def _halves(v):
    return v.half().view(torch.uint8).reshape(-1, 2)


def _weights(fmt, rows, cols, gen):
    """A packed tensor [rows, row bytes]: zero mean, standard deviation 1 / sqrt(cols)."""
    nb, std = rows * (cols // capi.BLK_ELEMS[FMT[fmt]]), 1.0 / math.sqrt(cols)
    w = torch.randint(0, 256, (nb, capi.BLK_BYTES[FMT[fmt]]), dtype=torch.uint8, device="cuda", generator=gen)
    spread = torch.rand(nb, device="cuda", generator=gen) * 0.4 + 0.8
    if fmt == "Q4_K":   # d * sc * (q - 7.5): every min equals its scale, dmin = 7.5 d; scales 32..63, q uniform
        d = spread * (std / (47.5 * 4.61))
        sc = torch.randint(32, 64, (nb, 8), dtype=torch.uint8, device="cuda", generator=gen)
        lo, hi = sc[:, :4], sc[:, 4:]
        w[:, 0:2], w[:, 2:4] = _halves(d), _halves(d * 7.5)
        w[:, 4:8] = lo | ((hi >> 4) << 6)
        w[:, 8:12] = w[:, 4:8]
        w[:, 12:16] = (hi & 15) | ((hi & 15) << 4)
    elif fmt == "Q6_K":   # d * sc * (q - 32), q uniform on 0..63, |sc| 64..127 with either sign
        sc = torch.randint(64, 128, (nb, 16), dtype=torch.int16, device="cuda", generator=gen)
        sign = torch.randint(0, 2, (nb, 16), dtype=torch.int16, device="cuda", generator=gen) * 2 - 1
        w[:, 192:208] = (sc * sign).to(torch.int8).view(torch.uint8)
        w[:, 208:210] = _halves(spread * (std / (97.0 * 18.5)))
    else:   # Q8_0: d * q
        w[:, 0:2] = _halves(spread * (std / 73.9))
    return w.reshape(rows, -1)


class _DeviceArray:
    """A view of device memory that the library owns; `owner` lives as long as a tensor made from it."""

    def __init__(self, owner, ptr, shape, strides):
        self.owner = owner
        self.__cuda_array_interface__ = {"data": (ptr, False), "shape": shape, "typestr": "<f2", "version": 3,
                                         "strides": tuple(2 * s for s in strides)}


def _view(owner, ptr, shape, strides):
    return torch.as_tensor(_DeviceArray(owner, ptr, tuple(shape), tuple(strides)), device="cuda")


def _fill_cache(dec, k_ptr, v_ptr, n_kv, max_kv, n_pos, gen):
    for ptr in (k_ptr, v_ptr):
        cache = _view(dec, ptr, (n_kv, n_pos, HEAD_DIM), (max_kv * HEAD_DIM, HEAD_DIM, 1))
        cache.copy_(torch.randn((n_kv, n_pos, HEAD_DIM), dtype=torch.float16, device="cuda", generator=gen))


def _seq_lengths(case):
    """Serving: the sequences are at different places, from a quarter of `pos` up to it."""
    n = case["n_seq"]
    return [max(1, case["pos"] * (n + 3 * (i + 1)) // (4 * n)) for i in range(n)]


def _decoder(case, gen, room):
    ctx, recipe = _context(), RECIPES[case["recipe"]]
    E, F, V, kv = case["n_embd"], case["n_ff"], case["n_vocab"], case["n_kv_head"]
    max_kv = (case["pos"] + room + 63) // 64 * 64
    cfg = dict(n_layer=case["n_layer"], n_embd=E, n_head=4 * kv, n_kv_head=kv, head_dim=HEAD_DIM, n_ff=F, n_vocab=V,
               max_kv=max_kv, rope_base=case["rope_base"], eps=1e-5)
    dec = Decoder(ctx, cfg)
    QD, KD, n_expert = 4 * kv * HEAD_DIM, kv * HEAD_DIM, case.get("n_expert", 0)
    shape = {"wq": (QD, E), "wk": (KD, E), "wv": (KD, E), "wo": (E, QD), "gate": (F, E), "up": (F, E), "down": (E, F)}

    def norm():
        return torch.rand(E, device="cuda", generator=gen) * 0.2 + 0.9

    for l in range(case["n_layer"]):
        for i, name in enumerate(LAYER):
            if n_expert and name in ("gate", "up", "down"):
                continue
            dec.set_layer_tensor(l, i, FMT[recipe[name]], _weights(recipe[name], *shape[name], gen))
        if n_expert:
            dec.set_layer_moe(l, _moe_block(case, gen, "Q4_K", 16))
        dec.set_layer_norms(l, norm(), norm())
    dec.set_global(capi.G_TOK_EMBD, FMT[recipe["tok_embd"]], _weights(recipe["tok_embd"], V, E, gen))
    dec.set_global(capi.G_OUTPUT, FMT[recipe["output"]], _weights(recipe["output"], V, E, gen))
    dec.set_out_norm(norm())
    return dec, max_kv


def _moe_block(case, gen, fmt, max_tokens):
    E, F, n = case["n_embd"], case["n_ff"], case["n_expert"]
    blk = MoeBlock(_context(), E, F, n, case["top_k"], norm=1, scale=1.0, fmt_gate_up=FMT[fmt], fmt_down=FMT[fmt],
                   max_tokens=max_tokens)
    router = torch.randn((n, E), device="cuda", generator=gen) * 0.02
    blk.set_weights(router, _weights(fmt, n * F, E, gen), _weights(fmt, n * F, E, gen), _weights(fmt, n * E, F, gen))
    return blk


def _rows_of(dec, ptrs, n_kv, max_kv, first, count):
    """The cache rows a pass appends. A pass hands back at most 60 of them: the deepest layers', which depend on the rest."""
    return [_view(dec, p + 2 * first * HEAD_DIM, (n_kv, count, HEAD_DIM), (max_kv * HEAD_DIM, HEAD_DIM, 1)) for p in ptrs][-60:]


def prepare(case, seed):
    gen, kind = _gen(seed), case["kind"]
    rng = random.Random(int(seed))
    s = {"case": case, "ctx": _context()}
    if kind == "matvec":
        s["w"] = _weights(case["fmt"], case["rows"], case["cols"], gen)
        s["x"] = torch.randn((case["nx"], case["cols"]), device="cuda", generator=gen)
        s["y"] = torch.zeros((case["nx"], case["rows"]), device="cuda")
    elif kind == "attention":
        B, kv, L = case["batch"], case["n_kv_head"], case["kv_len"]
        s["q"] = torch.randn((B, 4 * kv, HEAD_DIM), device="cuda", generator=gen)
        s["k"], s["v"] = (torch.randn((B, kv, L, HEAD_DIM), dtype=torch.float16, device="cuda", generator=gen) for _ in "kv")
        s["out"] = torch.zeros_like(s["q"])
    elif kind == "moe":
        s["moe"] = _moe_block(case, gen, case["fmt"], 16)
        s["x"] = torch.randn((case["n_tok"], case["n_embd"]), device="cuda", generator=gen)
        s["y"] = torch.zeros_like(s["x"])
    else:
        count = {"step": case.get("n_step"), "batch": case.get("m"), "seqs": 1}[kind]
        dec, max_kv = _decoder(case, gen, count)
        kv = case["n_kv_head"]
        s["dec"] = dec
        if kind == "seqs":
            dec.seqs_init(case["n_seq"])
            s["pos"], s["rows"] = _seq_lengths(case), []
            for l in range(case["n_layer"]):
                for i, p in enumerate(s["pos"]):
                    ptrs = dec.seqs_kv_ptrs(l, i)
                    _fill_cache(dec, *ptrs, kv, max_kv, p, gen)
                    s["rows"] += _rows_of(dec, ptrs, kv, max_kv, p, 1)
            s["rows"] = s["rows"][-60:]
            s["tokens"] = [rng.randrange(case["n_vocab"]) for _ in range(case["n_seq"])]
        else:
            ptrs = [dec.kv_ptrs(l) for l in range(case["n_layer"])]
            for p in ptrs:
                _fill_cache(dec, *p, kv, max_kv, case["pos"], gen)
            s["rows"] = _rows_of(dec, [x for p in ptrs for x in p], kv, max_kv, case["pos"], count)
            s["tokens"] = [rng.randrange(case["n_vocab"]) for _ in range(count)]
        dec.finalize()
    torch.cuda.synchronize()
    return s


def run(s):
    case, ctx = s["case"], s["ctx"]
    kind = case["kind"]
    if kind == "matvec":   # STREAM_DOT accumulates; a program zeroes its slots once per run
        y, nx, rows, cols = s["y"], case["nx"], case["rows"], case["cols"]
        if nx == 1:
            ctx.matvec_assign(FMT[case["fmt"]], s["w"], rows, cols, s["x"], y)
        else:
            capi._ck(ctx.lib.fl_b200_memset(ctx._h, C.c_void_p(y.data_ptr()), 0, C.c_size_t(4 * nx * rows)))
            ctx.matvec(FMT[case["fmt"]], s["w"], rows, cols, s["x"], y, nx=nx, xstride=cols, ystride=rows)
        return y
    if kind == "attention":
        ctx.attn_decode(s["q"], s["k"], s["v"], 4 * case["n_kv_head"], case["n_kv_head"], HEAD_DIM, case["kv_len"],
                        case["kv_len"], case["batch"], 1.0 / math.sqrt(HEAD_DIM), s["out"])
        return s["out"]
    if kind == "moe":
        s["moe"].forward(s["x"], case["n_tok"], s["y"])
        return s["y"]
    dec = s["dec"]
    if kind == "step":
        dec.rewind_to(case["pos"])
        tokens, tok = [], s["tokens"][0]
        for _ in range(case["n_step"]):
            tok = dec.step(tok)
            tokens.append(tok)
        return {"tokens": torch.tensor(tokens), "margin": dec.last_margin(), "logits": dec.logits(), "rows": s["rows"]}
    if kind == "batch":
        dec.rewind_to(case["pos"])
        tokens, margins = dec.step_batch(s["tokens"])
        last = case["m"] - 1
    else:
        for i, p in enumerate(s["pos"]):
            dec.seqs_set_pos(i, p)
        tokens, margins = dec.seqs_step(s["tokens"])
        last = case["n_seq"] - 1
    return {"tokens": torch.tensor(tokens), "margins": torch.tensor(margins), "logits": dec.batch_logits(last), "rows": s["rows"]}


# ---- what a pass cannot do without -------------------------------------------------------------------------------

def _tensor(fmt, rows, cols):
    return rows * capi.row_bytes(FMT[fmt], cols)


def _model_work(case, n_tok, keys, shared):
    """n_tok tokens through the model in one pass. keys: cached positions attended, summed over the tokens; shared: the
    tokens read one cache, else every token its own."""
    r, E, F, V = RECIPES[case["recipe"]], case["n_embd"], case["n_ff"], case["n_vocab"]
    QD, KD, n = 4 * case["n_kv_head"] * HEAD_DIM, case["n_kv_head"] * HEAD_DIM, case["n_layer"]
    layer = _tensor(r["wq"], QD, E) + _tensor(r["wk"], KD, E) + _tensor(r["wv"], KD, E) + _tensor(r["wo"], E, QD)
    macs = E * (2 * QD + 2 * KD)
    if case.get("n_expert"):
        expert = 2 * _tensor("Q4_K", F, E) + _tensor("Q4_K", E, F)
        layer += 4 * case["n_expert"] * E + expert * min(case["n_expert"], case["top_k"] * n_tok)
        macs += case["top_k"] * 3 * E * F + case["n_expert"] * E
    else:
        layer += _tensor(r["gate"], F, E) + _tensor(r["up"], F, E) + _tensor(r["down"], E, F)
        macs += 3 * E * F
    read = (keys // n_tok if shared else keys) * 2 * KD * 2
    weights = n * (layer + 8 * E) + _tensor(r["output"], V, E) + 4 * E
    return {"bytes": weights + n * (read + n_tok * 2 * KD * 2) + 4 * V * n_tok,
            "flops": 2 * (n_tok * (n * macs + V * E) + n * keys * 2 * QD)}


def work(case):
    kind = case["kind"]
    if kind == "matvec":
        rows, cols, nx = case["rows"], case["cols"], case["nx"]
        return {"bytes": _tensor(case["fmt"], rows, cols) + 4 * nx * (rows + cols), "flops": 2 * nx * rows * cols}
    if kind == "attention":
        B, kv, L = case["batch"], case["n_kv_head"], case["kv_len"]
        return {"bytes": B * kv * (4 * L * HEAD_DIM + 2 * 4 * 4 * HEAD_DIM), "flops": 2 * B * 4 * kv * L * HEAD_DIM * 2}
    if kind == "moe":
        E, F, n, T, k = case["n_embd"], case["n_ff"], case["n_expert"], case["n_tok"], min(case["top_k"], case["n_expert"])
        hit = n * (1 - (1 - k / n) ** T)   # expected number of experts that some token chose
        return {"bytes": hit * (2 * _tensor(case["fmt"], F, E) + _tensor(case["fmt"], E, F)) + 4 * n * E + 8 * T * E,
                "flops": 2 * T * (k * 3 * E * F + n * E)}
    if kind == "step":
        one = [_model_work(case, 1, case["pos"] + i + 1, True) for i in range(case["n_step"])]
        return {k: sum(w[k] for w in one) for k in ("bytes", "flops")}
    if kind == "batch":
        m = case["m"]
        return _model_work(case, m, sum(case["pos"] + i + 1 for i in range(m)), True)
    return _model_work(case, case["n_seq"], sum(p + 1 for p in _seq_lengths(case)), False)


def tolerance(case):
    """Four times what was measured. Operators against the same in 64 bits: relative error 1 .. 6e-7 (32-bit sums, 22-bit
    activations; largest single error 2.8e-6 of the value), attention 2.2e-6 at 64K keys (7.1e-6). Whole models against
    themselves with other sums (f16 instead of integer arithmetic, single steps instead of a batch pass): logits 4e-7 ..
    5.1e-5, margins, which are small differences of logits, 1.1e-4, cache rows 1.1e-6: the f32 differences flip f16
    roundings of cache rows."""
    if case["kind"] in ("matvec", "moe"):
        return {"rel": 3e-6, "max": 2e-5}
    if case["kind"] == "attention":
        return {"rel": 1e-5, "max": 4e-5}
    return {"rel": 5e-4, "max": 5e-3}
