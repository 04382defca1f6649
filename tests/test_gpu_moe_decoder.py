"""GPU parity tests of a decoder with mixture-of-experts layers (Mixtral shape: attention as in the dense
model, the feed-forward block replaced by router -> top-k experts -> weighted merge; the chain the reference's graph
builder emits per MoE layer, src/model/decoder.cpp:925-1045) against the CPU oracle's step on identical weights."""
import numpy as np
import pytest

from fast_llm_b200 import capi, synth
from fast_llm_b200.decoder import Decoder
from fast_llm_b200.moe import MoeBlock
from test_gpu_decoder import build_pair, force_kv, logits_close, LOGIT_TOL, HIDDEN_TOL

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

# two MoE layers around a dense one; the query width equals n_embd (the block's output borrows the query buffer)
CFG = dict(n_layer=3, n_embd=2048, n_head=16, n_kv_head=4, head_dim=128, n_ff=4096, n_vocab=1000, max_kv=96,
           rope_base=500000.0, eps=1e-5)
MOE_LAYERS = (0, 2)
NE, K, F = 4, 2, 1024


def build_moe_pair(ctx, checker, seed, n_prefill, fmt_down=capi.Q4_K, max_tokens=8, fmt_gu=capi.Q4_K, NE=NE, K=K, F=F):
    """build_pair's dense model, then layers MOE_LAYERS get an expert block on both sides (their dense gate / up / down
    stay set on the oracle side and are simply not used there either)."""
    dec, orc = build_pair(ctx, checker, CFG, seed, n_prefill, finalize=False)
    blocks = []
    for l in MOE_LAYERS:
        rng = synth.rng_for(seed, "L%d.moe" % l)
        E = CFG["n_embd"]
        wg = synth.quant_tensor(fmt_gu, rng, NE * F, E); wu = synth.quant_tensor(fmt_gu, rng, NE * F, E)
        wd = synth.quant_tensor(fmt_down, rng, NE * E, F)
        wr = rng.standard_normal((NE, E)).astype(np.float32)     # wide logits: no near-ties between experts
        blk = MoeBlock(ctx, E, F, NE, K, norm=1, scale=1.0, fmt_gate_up=fmt_gu, fmt_down=fmt_down, max_tokens=max_tokens)
        blk.set_weights(*(torch.from_numpy(np.ascontiguousarray(a)).cuda() for a in (wr, wg, wu, wd)))
        dec.set_layer_moe(l, blk)
        orc.set_layer_moe(l, NE, K, 1, 1.0, F, wr, fmt_gu, wg, wu, fmt_down, wd)
        blocks.append(blk)
    torch.cuda.synchronize()
    dec.finalize()
    dec.rewind_to(n_prefill)
    orc.set_n_past(n_prefill)
    return dec, orc, blocks


@pytest.mark.parametrize("fmt_down", [capi.Q4_K, capi.Q6_K])
def test_moe_model_teacher_forced(ctx, checker, fmt_down):
    dec, orc, blocks = build_moe_pair(ctx, checker, seed=11, n_prefill=30, fmt_down=fmt_down)
    tok = 7
    for step in range(8):
        want_tok = orc.step(tok)
        got_tok = dec.step(tok)
        got, want = dec.logits(), orc.logits()
        assert np.all(np.isfinite(got)) and ctx.status() == 0
        err = logits_close(got, want)
        assert err < LOGIT_TOL, (step, err)
        if got_tok != want_tok:
            assert orc.margin() <= 2 * np.max(np.abs(got - want)), (step, got_tok, want_tok, orc.margin())
        assert logits_close(dec.tap(0), orc.hidden()) < HIDDEN_TOL
        # the last MoE layer routed to the experts the oracle chose
        ids, gates = blocks[-1].routing(1)
        assert sorted(ids[0]) == sorted(int(i) for i in np.ctypeslib.as_array(orc.p.flo_llama_moe_ids(orc.h), shape=(K,)))
        force_kv(ctx, dec, orc, CFG, 30 + step)
        tok = want_tok
    # the step's bytes: attention tensors of every layer, dense FFN of layer 1, router + K experts of the MoE layers
    wb, _ = dec.bytes_per_step(30)
    E, QD, KD = CFG["n_embd"], CFG["n_head"] * 128, CFG["n_kv_head"] * 128
    rb = capi.row_bytes
    attn = QD * rb(capi.Q4_K, E) + KD * rb(capi.Q4_K, E) + KD * rb(capi.Q6_K, E) + E * rb(capi.Q4_K, QD) + 2 * E * 4
    dense = 2 * CFG["n_ff"] * rb(capi.Q4_K, E) + E * rb(capi.Q6_K, CFG["n_ff"])
    moe = NE * E * 4 + K * (2 * F * rb(capi.Q4_K, E) + E * rb(fmt_down, F))
    assert wb == 3 * attn + dense + 2 * moe + CFG["n_vocab"] * rb(capi.Q6_K, E) + E * 4
    dec.close(); orc.close()


def test_moe_model_run_and_batch_pass(ctx, checker):
    """Device feedback equals step-by-step calls; the batch pass (every expert once for the tokens that chose it)
    gives the tokens of single steps."""
    dec, orc, _ = build_moe_pair(ctx, checker, seed=13, n_prefill=12)
    toks = [int(t) for t in dec.run(3, 6)]
    dec.rewind_to(12)
    t, seq = 3, []
    for _ in range(6):
        t = dec.step(t)
        seq.append(t)
    assert toks == seq
    dec.rewind_to(12)
    outs, margins = dec.step_batch([3] + seq[:5])          # teacher-forced inputs: 3, a0 .. a4
    for i, (o, mg) in enumerate(zip(outs, margins)):
        assert o == seq[i] or mg < 1e-2, (i, o, seq[i], mg)
    dec.close(); orc.close()


# one token: all slots' experts in one launch for gate | up and one for down (csrc/matvec_expert.cu). Columns of a part segment, of
# one, of the most blocks a thread converts at once and of more; one slot, as many slots as experts; units that leave groups and
# CTAs without work; the last shape is not taken (Q6_K rows of 1024 columns are no whole 16 bytes).
@pytest.mark.parametrize("fmt_gu,fmt_down,NE,K,F", [
    (capi.Q4_K, capi.Q4_K, 4, 1, 512), (capi.Q4_K, capi.Q4_K, 8, 3, 2304), (capi.Q6_K, capi.Q6_K, 3, 3, 2048),
    (capi.Q4_K, capi.Q6_K, 2, 2, 10240), (capi.Q6_K, capi.Q4_K, 4, 2, 9216), (capi.Q4_K, capi.Q4_K, 2, 1, 18432), (capi.Q4_K, capi.Q6_K, 4, 2, 1024)])
def test_one_token_over_its_experts(ctx, checker, fmt_gu, fmt_down, NE, K, F):
    dec, orc, blocks = build_moe_pair(ctx, checker, 17, 5, fmt_down, 4, fmt_gu, NE, K, F)
    tok = 7
    for step in range(2):
        want_tok = orc.step(tok)
        got_tok = dec.step(tok)
        got, want = dec.logits(), orc.logits()
        assert np.all(np.isfinite(got)) and ctx.status() == 0
        assert logits_close(got, want) < LOGIT_TOL
        if got_tok != want_tok:
            assert orc.margin() <= 2 * np.max(np.abs(got - want))
        assert logits_close(dec.tap(0), orc.hidden()) < HIDDEN_TOL
        ids, gates = blocks[-1].routing(1)
        assert sorted(ids[0]) == sorted(int(i) for i in np.ctypeslib.as_array(orc.p.flo_llama_moe_ids(orc.h), shape=(K,)))
        force_kv(ctx, dec, orc, CFG, 5 + step)
        tok = want_tok
    dec.close(); orc.close()


def gpu_decoder(ctx, E, F, NE, K, fmt_gu, fmt_down, seed, spoil=None):
    """One layer of attention and experts over random weights, without an oracle. spoil(gate): last change of the gate rows."""
    gen = torch.Generator(device="cuda").manual_seed(seed)

    def quants(fmt, rows, cols):
        n = rows * cols // capi.BLK_ELEMS[fmt]
        w = torch.randint(0, 256, (n, capi.BLK_BYTES[fmt]), dtype=torch.uint8, device="cuda", generator=gen)
        d = ((torch.rand(n, device="cuda", generator=gen) * 0.4 + 0.8) / (cols ** 0.5 * 400)).half().view(torch.uint8).reshape(-1, 2)
        for o in {capi.Q4_K: (0, 2), capi.Q6_K: (208,)}[fmt]:
            w[:, o:o + 2] = d
        return w.reshape(rows, -1)

    def norm():
        return torch.rand(E, device="cuda", generator=gen) * 0.2 + 0.9

    kv = E // 512
    dec = Decoder(ctx, dict(n_layer=1, n_embd=E, n_head=4 * kv, n_kv_head=kv, head_dim=128, n_ff=512, n_vocab=600, max_kv=64, rope_base=1e4, eps=1e-5))
    for i, (r, c) in enumerate(((E, E), (E // 4, E), (E // 4, E), (E, E))):
        dec.set_layer_tensor(0, i, capi.Q4_K, quants(capi.Q4_K, r, c))
    blk = MoeBlock(ctx, E, F, NE, K, fmt_gate_up=fmt_gu, fmt_down=fmt_down, max_tokens=1)
    gate = quants(fmt_gu, NE * F, E)
    if spoil:
        spoil(gate)
    blk.set_weights(torch.randn((NE, E), device="cuda", generator=gen), gate, quants(fmt_gu, NE * F, E), quants(fmt_down, NE * E, F))
    dec.set_layer_moe(0, blk)
    dec.set_layer_norms(0, norm(), norm())
    dec.set_global(capi.G_TOK_EMBD, capi.Q4_K, quants(capi.Q4_K, 600, E))
    dec.set_global(capi.G_OUTPUT, capi.Q4_K, quants(capi.Q4_K, 600, E))
    dec.set_out_norm(norm())
    torch.cuda.synchronize()
    dec.finalize()
    return dec


@pytest.mark.parametrize("fmt", [capi.Q4_K, capi.Q6_K])
def test_a_token_hides_no_nan(ctx, fmt):
    """A NaN in one row's result of gate reaches the whole output of the block through down, and the logits."""
    E, F, NE = 2048, 2048, 4

    def spoil(gate):   # the scale of the first block of row 100 of every expert
        at = {capi.Q4_K: 0, capi.Q6_K: 208}[fmt]
        gate.view(NE, F, -1)[:, 100, at:at + 2] = torch.tensor([0x00, 0x7e], dtype=torch.uint8, device="cuda")

    dec = gpu_decoder(ctx, E, F, NE, 2, fmt, fmt, 5, spoil)
    dec.step(7)
    assert np.isnan(dec.logits()).all()
    dec.close()


@pytest.mark.parametrize("E,fmt_gu,fmt_down,NE,K,F", [
    (2048, capi.Q4_K, capi.Q4_K, 4, 1, 512), (2048, capi.Q4_K, capi.Q6_K, 8, 3, 2048), (2048, capi.Q6_K, capi.Q4_K, 3, 3, 2304),
    (4096, capi.Q4_K, capi.Q4_K, 4, 2, 14336), (4096, capi.Q6_K, capi.Q6_K, 4, 2, 10240), (6144, capi.Q4_K, capi.Q6_K, 2, 2, 4096),
    (6144, capi.Q6_K, capi.Q4_K, 4, 2, 9216), (8192, capi.Q4_K, capi.Q4_K, 2, 2, 2048)])
def test_a_token_has_the_bits_of_a_launch_per_slot(ctx, monkeypatch, E, fmt_gu, fmt_down, NE, K, F):
    """The selected experts in two launches (csrc/matvec_expert.cu) against a launch of the streaming kernel per slot: the same 21-bit
    activations, exact integer sums and order of f32 sums, hence the same bits, up to 6144 columns of gate and up; above, the sum of squares
    of the norm is taken in another order (16 units of 2^-24 at most between any two orders of so many warps, the logits 2e-6 measured)."""
    seen = {}
    for form in ("1", "0"):
        monkeypatch.setenv("FLB_MOE_TOKEN", form)
        dec = gpu_decoder(ctx, E, F, NE, K, fmt_gu, fmt_down, 11)
        steps, tok = [], 5
        for _ in range(3):
            dec.step(tok)
            steps.append((dec.logits().copy(), dec.tap(0).copy()))
            tok += 101
        assert all(np.isfinite(v).all() for s in steps for v in s) and ctx.status() == 0
        seen[form] = steps, dec.launches_per_step()
        dec.close()
    (a, launches), (b, per_slot) = seen["1"], seen["0"]
    assert per_slot - launches == (1 + 2 * K + 1) - 4    # router, then gate | up and down once or per slot, merge
    for (la, ha), (lb, hb) in zip(a, b):
        if E <= 6144:
            assert np.array_equal(la, lb) and np.array_equal(ha, hb)
        else:
            assert np.linalg.norm(la - lb) <= 1e-5 * np.linalg.norm(lb) and np.linalg.norm(ha - hb) <= 1e-5 * np.linalg.norm(hb)
