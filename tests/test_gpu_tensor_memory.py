"""GPU tests of the multi-column matmul with the weights in tensor memory (csrc/matmul_tm.cu): by itself (FLB_UMMA=1 sends every
Q4_K call of several columns there) at the edges of its tiles of 128 rows, steps of 256 columns and 8 / 16 tokens, and with its planes
of partial sums in a batch pass whose FFN is large enough for it.

Tolerance of a matmul as in test_gpu_multi_column.py (the sums are the same): 1e-5 of the root mean square of the exact result.
Batch passes against single steps as in test_gpu_batch_forms.py: 5e-4 of the logits."""
import numpy as np
import pytest

from fast_llm_b200 import capi, synth

pytestmark = pytest.mark.gpu
torch = pytest.importorskip("torch")


@pytest.mark.parametrize("rows,cols,nx", [
    (1, 256, 2), (127, 512, 8), (128, 768, 9), (129, 2304, 16), (300, 4096, 5), (64, 18432, 16), (37, 14336, 33),
    (20000, 256, 7),       # more tiles than CTAs, one step each
    (148 * 128, 1024, 16), (148 * 128 + 1, 1024, 3),
])
def test_whole_tiles(ctx, monkeypatch, rows, cols, nx):
    monkeypatch.setenv("FLB_UMMA", "1")
    w = torch.from_numpy(synth.quant_tensor(capi.Q4_K, np.random.default_rng(rows + cols), rows, cols)).cuda()
    f = torch.empty((rows, cols), device="cuda")
    gen = torch.Generator(device="cuda").manual_seed(nx)
    x = torch.full((nx, cols + 8), float("nan"), device="cuda")   # the gap between columns is never read
    x[:, :cols] = torch.randn((nx, cols), device="cuda", generator=gen) * torch.logspace(-3, 3, nx, device="cuda")[:, None]
    y = torch.randn((nx, rows + 3), device="cuda", generator=gen)
    torch.cuda.synchronize()
    ctx.dequant(capi.Q4_K, w, rows, cols, f)
    ctx.sync()
    want = y.double()
    want[:, :rows] += x[:, :cols].double() @ f.double().T
    torch.cuda.synchronize()
    ctx.matvec(capi.Q4_K, w, rows, cols, x, y, nx=nx, xstride=cols + 8, ystride=rows + 3)
    ctx.sync()
    assert ctx.status() == 0
    err = (y.double() - want)[:, :rows].abs().amax(1) / want[:, :rows].pow(2).mean(1).sqrt()
    assert float(err.max()) <= 1e-5
    assert torch.equal(y[:, rows:].double(), want[:, rows:])


@pytest.mark.parametrize("nx", [8, 16])
def test_launches_in_a_row(ctx, monkeypatch, nx):
    """Launches whose CTAs have one to five steps, one behind the other without a wait between them: a CTA waits for the last
    arrival at the barrier of either weight buffer (an odd number of steps leaves the second one phase behind, one step never
    uses it) before the next CTA sets up its own in the same memory. A wait on the wrong phase runs out and says so in the
    status; a missing one shows by reading only."""
    monkeypatch.setenv("FLB_UMMA", "1")
    rows, cols = 148 * 128, 256
    w = torch.from_numpy(synth.quant_tensor(capi.Q4_K, np.random.default_rng(nx), 5 * rows, cols)).cuda()
    f = torch.empty((5 * rows, cols), device="cuda")
    x = torch.randn((nx, cols), device="cuda", generator=torch.Generator(device="cuda").manual_seed(nx))
    ys = [torch.zeros((nx, k * rows), device="cuda") for k in range(1, 6)]
    torch.cuda.synchronize()
    ctx.dequant(capi.Q4_K, w, 5 * rows, cols, f)
    for _ in range(6):
        for k, y in enumerate(ys, 1):
            ctx.matvec(capi.Q4_K, w, k * rows, cols, x, y, nx=nx, xstride=cols, ystride=k * rows)
    ctx.sync()
    assert ctx.status() == 0
    want = 6 * (x.double() @ f.double().T)
    for k, y in enumerate(ys, 1):
        assert float((y.double() - want[:, :k * rows]).abs().max() / want.pow(2).mean().sqrt()) <= 1e-5, k


@pytest.mark.parametrize("m", [2, 4, 5, 8, 9, 16])
@pytest.mark.parametrize("recipe,n_embd,n_ff", [("Q4_K", 4096, 14336), ("Q4_K", 2048, 9472), ("Q4_K", 4096, 4864), ("Q4_K_M", 4096, 14336)])
def test_batch_pass(recipe, n_embd, n_ff, m):
    """Gate | up (two planes) and, where it is large enough, down (six planes): 9472 x 2 rows of 2048 columns are the fewest steps
    that 8 tokens take this form for, 4864 x 2 of 4096 leave tiles shared by three CTAs."""
    from perf import cases
    case = dict(kind="batch", pos=70, m=m, n_layer=1, n_embd=n_embd, n_kv_head=n_embd // 512, n_ff=n_ff, n_vocab=1000, recipe=recipe,
                rope_base=500000.0)
    s = cases.prepare(case, m)
    dec = s["dec"]
    dec.rewind_to(70)
    outs, margins = dec.step_batch(s["tokens"])
    got = [dec.batch_logits(i) for i in range(m)]
    dec.rewind_to(70)
    again, _ = dec.step_batch(s["tokens"])
    assert again == outs and all(np.array_equal(dec.batch_logits(i), got[i]) for i in range(m))
    dec.rewind_to(70)
    for i, t in enumerate(s["tokens"]):
        dec.step(t)
        single = dec.logits()
        assert np.linalg.norm(got[i] - single) / np.linalg.norm(single) <= 5e-4
        assert abs(margins[i] - dec.last_margin()) <= 2 * np.abs(got[i] - single).max() + 1e-6
    assert s["ctx"].status() == 0
    dec.close()
