"""GPU tests of the multi-column matmul with the weights in tensor memory (csrc/matmul_tm.cu): by itself, in whole tiles
(FLB_UMMA=1 sends every Q4_K call of several columns there) and in the shares and planes of partial sums that a batch pass uses
(FLB_UMMA=2, Q4_K and Q6_K), at the edges of its tiles of 128 rows, steps of 256 columns and 8 / 16 tokens; and in batch passes at
the edges of the rule that picks it.

Tolerance of a matmul as in test_gpu_multi_column.py (the sums are the same): 1e-5 of the root mean square of the exact result.
Batch passes against single steps as in test_gpu_batch_forms.py: 5e-4 of the logits."""
import numpy as np
import pytest

import test_gpu_multi_column as multi_column
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


@pytest.mark.parametrize("fmt,rows,cols,nx", [
    (capi.Q4_K, 1, 256, 2), (capi.Q4_K, 129, 768, 9), (capi.Q4_K, 20000, 256, 16),    # one block: a tile is one CTA's
    (capi.Q4_K, 28672, 4096, 8), (capi.Q4_K, 28672, 4096, 16), (capi.Q4_K, 300, 2304, 33),
    (capi.Q6_K, 100, 2048, 2), (capi.Q6_K, 4096, 14336, 8), (capi.Q6_K, 4096, 14336, 16), (capi.Q6_K, 12801, 2048, 5),
    (capi.Q4_K, 1024, 6144, 9), (capi.Q6_K, 1000, 6144, 3),                           # the most planes, 8
    (capi.Q4_K, 64, 18432, 16), (capi.Q6_K, 200, 18432, 8),                           # the most columns
    (capi.Q4_K, 131072, 4352, 16),                                                    # more rows than the planes hold: slices
])
def test_planes(ctx, monkeypatch, fmt, rows, cols, nx):
    """Shares that cut tiles anywhere. The memory of the planes holds NaN before: a plane that a tile has no sums for is cleared."""
    monkeypatch.setenv("FLB_UMMA", "2")
    w = torch.from_numpy(synth.quant_tensor(capi.Q4_K, np.random.default_rng(1), 65536, 256)).cuda()
    x, y = torch.full((16, 256), float("nan"), device="cuda"), torch.zeros((16, 65536), device="cuda")
    torch.cuda.synchronize()
    ctx.matvec(capi.Q4_K, w, 65536, 256, x, y, nx=16, xstride=256, ystride=65536)
    ctx.sync()
    assert torch.isnan(y).all()
    multi_column.test_multi_column_edges(ctx, fmt, rows, cols, nx)


@pytest.mark.parametrize("form,fmt", [("1", capi.Q4_K), ("2", capi.Q4_K), ("2", capi.Q6_K)])
def test_special_values(ctx, monkeypatch, form, fmt):
    monkeypatch.setenv("FLB_UMMA", form)
    multi_column.test_multi_column_special_values(ctx, fmt)


@pytest.mark.parametrize("form", ["0", "2"])
@pytest.mark.parametrize("nx", [8, 16])
def test_q6_k_smallest_and_largest_scales(ctx, monkeypatch, form, nx):
    """The block scales of weight and activation meet in the result only: their product alone may not be a finite or a normal
    number. Rows of scale zero under d = 40000 and an activation near the end of the range give zero; d of two bits in f16's
    last places times an activation of 1e-35 is as exact as any other."""
    monkeypatch.setenv("FLB_UMMA", form)
    rows, cols = 256, 2048
    w = torch.from_numpy(synth.quant_tensor(capi.Q6_K, np.random.default_rng(0), rows, cols)).cuda()
    blk = w.view(-1, 210)
    x = torch.randn((nx, cols), device="cuda", generator=torch.Generator(device="cuda").manual_seed(0))
    f = torch.empty((rows, cols), device="cuda")
    for d, size in ((40000.0, 1e37), (3 * 2.0 ** -24, 1e-35)):
        blk[:, 208:210] = torch.tensor([d], dtype=torch.float16, device="cuda").view(torch.uint8)
        xs, y = x * size, torch.zeros((nx, rows), device="cuda")
        xs[:, 5::256] = 8.9 * size                      # the largest of every block, the same block scale everywhere
        if d > 1:
            blk[:, 192:208] = 0
        else:
            blk[:, 192:208] = 100
        torch.cuda.synchronize()
        ctx.dequant(capi.Q6_K, w, rows, cols, f)
        ctx.matvec(capi.Q6_K, w, rows, cols, xs, y, nx=nx, xstride=cols, ystride=rows)
        ctx.sync()
        if d > 1:
            assert torch.equal(y, torch.zeros_like(y))
        else:
            assert multi_column.close(y, xs.double() @ f.double().T)


@pytest.mark.parametrize("rows,cols", [(4096, 4096), (4096, 14336)])
@pytest.mark.parametrize("nx", [2, 8, 9, 16])
@pytest.mark.parametrize("form,recipe", [("1", "Q4_K"), ("2", "Q4_K"), ("2", "Q6_K")])
def test_sums_are_not_truncated(ctx, monkeypatch, form, recipe, nx, rows, cols):
    """Bias and 2-norm of the error as test_gpu_multi_column.py asks them of the other kernel: tcgen05.mma truncates its running sum
    as mma.sync does, so that the chains are as short."""
    from perf import cases
    monkeypatch.setenv("FLB_UMMA", form)
    fmt = cases.FMT[recipe]
    gen = torch.Generator(device="cuda").manual_seed(nx)
    w = cases._weights(recipe, rows, cols, gen)
    f = torch.empty((rows, cols), device="cuda")
    x = torch.randn((nx, cols), device="cuda", generator=gen)
    y = torch.zeros((nx, rows), device="cuda")
    torch.cuda.synchronize()
    ctx.dequant(fmt, w, rows, cols, f)
    ctx.matvec(fmt, w, rows, cols, x, y, nx=nx, xstride=cols, ystride=rows)
    ctx.sync()
    want = x.double() @ f.double().T
    bias, err = float((y.double() * want).sum() / want.pow(2).sum()) - 1, float((y.double() - want).norm() / want.norm())
    assert abs(bias) <= 8e-8, bias
    assert err <= 1.5e-7, err


@pytest.mark.parametrize("rows,cols", [(4096, 4096), (2048, 14336), (2048, 18432)])
@pytest.mark.parametrize("nx", [4, 8, 16])
@pytest.mark.parametrize("recipe", ["Q4_K", "Q6_K"])
def test_no_less_exact_than_the_other_form(ctx, monkeypatch, recipe, nx, rows, cols):
    """Error against 64 bits (2-norm) of the shares that a pass uses and of matmul_nx_kernel on the same product. Of n > 8000 results,
    whose errors are independent, the 2-norm scatters by 1 / sqrt(2 n) < 0.8 % in either form: 2 % of room."""
    from perf import cases
    fmt, err = cases.FMT[recipe], {}
    gen = torch.Generator(device="cuda").manual_seed(nx)
    w, f = cases._weights(recipe, rows, cols, gen), torch.empty((rows, cols), device="cuda")
    x = torch.randn((nx, cols), device="cuda", generator=gen)
    torch.cuda.synchronize()
    ctx.dequant(fmt, w, rows, cols, f)
    ctx.sync()
    want = x.double() @ f.double().T
    for form in "02":
        monkeypatch.setenv("FLB_UMMA", form)
        y = torch.zeros((nx, rows), device="cuda")
        torch.cuda.synchronize()
        ctx.matvec(fmt, w, rows, cols, x, y, nx=nx, xstride=cols, ystride=rows)
        ctx.sync()
        err[form] = float((y.double() - want).norm() / want.norm())
    assert err["2"] <= 1.02 * err["0"], err


@pytest.mark.parametrize("nx", [8, 16])
def test_launches_in_a_row(ctx, monkeypatch, nx):
    """Launches whose CTAs have one to five steps, one behind the other without a wait between them: after the last step of either
    weight buffer nothing arrives at its barrier any more, so that the next CTA can set up its own in the same memory. One arrival
    too few and a wait runs out, which the status says; one too many shows by reading only."""
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


@pytest.mark.parametrize("recipe,n_embd,n_ff,m,taken", [
    ("Q4_K_M", 4096, 14336, 2, True), ("Q4_K_M", 4096, 14336, 8, True), ("Q4_K_M", 4096, 10240, 5, True),   # Q6_K down with few tokens
    ("Q4_K_M", 4096, 4096, 9, True), ("Q4_K_M", 4096, 4096, 16, True), ("Q4_K_M", 4096, 4096, 8, False),     # O and down, from 9 on
    ("Q4_K", 2048, 9472, 8, True), ("Q4_K", 2048, 9216, 8, False),   # 8 and 7.8 steps per CTA in gate | up
    ("Q4_K", 1024, 7168, 9, True), ("Q4_K", 1024, 6912, 9, False),   # 3.03 and 2.9
])
def test_pass_with_and_without(monkeypatch, recipe, n_embd, n_ff, m, taken):
    """The pass against itself with FLB_UMMA=0, on a layer whose Q, K and V go the same way in both: K and V are then the same
    bits and no flipped f16 rounding covers anything, so that 1 / rms per token, the planes and both formats show as sums in another
    order. O (from 9 tokens on), gate, up, down and the head, whose input then differs, are each 1.3e-7 off (2-norm) in either
    form, independently: sqrt(10) of that is 4.1e-7, and a tenth more for the scatter from token to token (measured 3.7e-7). Launches
    that the rule leaves to the other kernel: the same bits."""
    from perf import cases
    case = dict(kind="batch", pos=70, m=m, n_layer=1, n_embd=n_embd, n_kv_head=n_embd // 512, n_ff=n_ff, n_vocab=1000, recipe=recipe,
                rope_base=500000.0)
    logits = []
    for off in (False, True):
        if off:
            monkeypatch.setenv("FLB_UMMA", "0")
        s = cases.prepare(case, m)
        s["dec"].rewind_to(70)
        s["dec"].step_batch(s["tokens"])
        logits.append(np.stack([s["dec"].batch_logits(i) for i in range(m)]).astype(np.float64))
        assert s["ctx"].status() == 0
        s["dec"].close()
    diff = np.linalg.norm(logits[0] - logits[1], axis=1) / np.linalg.norm(logits[1], axis=1)
    assert (diff.max() > 0) == taken
    assert diff.max() <= 4.5e-7, diff


@pytest.mark.parametrize("recipe,n_embd,n_vocab,m,taken", [
    ("Q4_K", 1024, 75776, 9, True), ("Q4_K", 1024, 75776, 8, False), ("Q4_K", 1024, 75649, 16, True), ("Q4_K", 1024, 75648, 16, False),
    ("Q4_K_M", 2048, 75777, 9, True), ("Q4_K_M", 2048, 80000, 16, True)])
def test_head_of_a_pass(monkeypatch, recipe, n_embd, n_vocab, m, taken):
    """The head in whole tiles, four rounds of them at least (592 tiles on 148 SMs), the last one ragged: the pass against itself with
    FLB_UMMA=0 on a model whose other matmuls are too small for this form. The head alone differs, each form 1.3e-7 off (2-norm),
    independently: 1.9e-7, and a third more for the scatter from token to token."""
    from perf import cases
    case = dict(kind="batch", pos=20, m=m, n_layer=1, n_embd=n_embd, n_kv_head=n_embd // 512, n_ff=2048, n_vocab=n_vocab, recipe=recipe,
                rope_base=500000.0)
    logits, tokens = [], []
    for off in (False, True):
        if off:
            monkeypatch.setenv("FLB_UMMA", "0")
        s = cases.prepare(case, m)
        s["dec"].rewind_to(20)
        tokens.append(s["dec"].step_batch(s["tokens"])[0])
        logits.append(np.stack([s["dec"].batch_logits(i) for i in range(m)]).astype(np.float64))
        assert s["ctx"].status() == 0
        s["dec"].close()
    diff = np.linalg.norm(logits[0] - logits[1], axis=1) / np.linalg.norm(logits[1], axis=1)
    assert np.isfinite(logits[0]).all() and (diff.max() > 0) == taken
    assert diff.max() <= 2.5e-7, diff
    assert [int(np.argmax(l)) for l in logits[0]] == list(tokens[0])
