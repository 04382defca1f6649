"""GPU tests of the forms of the batch pass (Decoder.step_batch, Decoder.seqs_step) that the Q4_K_M models of the other tests
do not reach, against the same tokens as single steps: tensor by tensor (a width the multi-column kernel does not take;
FLB_UMMA=1), every tensor in Q8_0, and three formats side by side in one launch.

Weights of zero mean and standard deviation 1 / sqrt(columns) keep activations at unit size, so that the f32 differences
between the forms show as flipped f16 roundings of single cache values (2^-11 of a value): logits up to 1.8e-4 apart in the 2-norm,
measured; the bound is 5e-4, a wrong tensor, position or scale is far above it."""
import numpy as np
import pytest

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")

MODEL = dict(n_layer=2, n_embd=2048, n_kv_head=4, n_ff=4096, n_vocab=1000, rope_base=500000.0)
MIXED = {"wq": "Q4_K", "wk": "Q6_K", "wv": "Q8_0", "wo": "Q8_0", "gate": "Q6_K", "up": "Q4_K", "down": "Q4_K", "output": "Q8_0",
         "tok_embd": "Q6_K"}
FORMS = {
    "wide_q8_0": dict(MODEL, n_ff=18688, recipe="Q8_0"),   # more columns than the multi-column kernel takes
    "wide_q4_k": dict(MODEL, n_ff=18688, recipe="Q4_K"),
    "tcgen05": dict(MODEL, recipe="Q4_K"),                 # with FLB_UMMA=1
    "q8_0": dict(MODEL, recipe="Q8_0"),
    "mixed": dict(MODEL, recipe="mixed"),
}


@pytest.fixture
def cases(monkeypatch):
    from perf import cases
    monkeypatch.setitem(cases.RECIPES, "mixed", MIXED)
    return cases


def check(dec, got, margin, tok, single):
    err = np.linalg.norm(got - single) / np.linalg.norm(single)
    assert err <= 5e-4, err
    assert abs(margin - dec.last_margin()) <= 2 * np.abs(got - single).max() + 1e-6
    if tok != int(single.argmax()):
        assert dec.last_margin() <= 2 * np.abs(got - single).max()


@pytest.mark.parametrize("m", [2, 3, 4, 8, 9, 16])
@pytest.mark.parametrize("form", FORMS)
def test_batch_pass_equals_single_steps(cases, monkeypatch, form, m):
    if form == "tcgen05":
        monkeypatch.setenv("FLB_UMMA", "1")
    s = cases.prepare(dict(kind="batch", pos=70, m=m, **FORMS[form]), m)
    dec = s["dec"]
    dec.rewind_to(70)
    outs, margins = dec.step_batch(s["tokens"])
    got = [dec.batch_logits(i) for i in range(m)]
    dec.rewind_to(70)
    for i, t in enumerate(s["tokens"]):
        dec.step(t)
        check(dec, got[i], margins[i], outs[i], dec.logits())
    assert s["ctx"].status() == 0
    dec.close()


@pytest.mark.parametrize("n_seq", [2, 8, 9, 16])
@pytest.mark.parametrize("form", FORMS)
def test_sequences_equal_single_steps(cases, monkeypatch, form, n_seq):
    """Three tokens each from an empty cache."""
    if form == "tcgen05":
        monkeypatch.setenv("FLB_UMMA", "1")
    s = cases.prepare(dict(kind="seqs", pos=64, n_seq=n_seq, **FORMS[form]), n_seq)
    dec = s["dec"]
    toks = np.random.default_rng(n_seq).integers(0, MODEL["n_vocab"], (3, n_seq))
    for i in range(n_seq):
        dec.seqs_set_pos(i, 0)
    got = []
    for row in toks:
        outs, margins = dec.seqs_step([int(t) for t in row])
        got.append((outs, margins, [dec.batch_logits(i) for i in range(n_seq)]))
    for i in range(n_seq):
        dec.rewind_to(0)
        for step, (outs, margins, logits) in enumerate(got):
            dec.step(int(toks[step, i]))
            check(dec, logits[i], margins[i], outs[i], dec.logits())
    assert s["ctx"].status() == 0
    dec.close()
